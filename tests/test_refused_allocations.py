"""What the host side leaves behind when an allocation is refused (no device needed)."""
from host_program import compile_and_run


def test_staged_tile_layout_is_whole_or_absent(tmp_path):
    assert "refused in turn" in compile_and_run("brick_layout", tmp_path)
