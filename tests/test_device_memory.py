"""What the host side holds on the device, and what it leaves when an allocation is refused (no
device needed)."""
from host_program import compile_and_run


def test_staged_tile_layout_is_whole_or_absent(tmp_path):
    assert "refused in turn" in compile_and_run("brick_layout", tmp_path)


def test_sample_list_is_as_long_as_its_samples(tmp_path):
    assert "1 samples" in compile_and_run("sample_list", tmp_path)


def test_what_a_context_keeps_goes_back(tmp_path):
    assert "went back" in compile_and_run("kept_memory", tmp_path)
