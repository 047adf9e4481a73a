"""Images whose device address is given out: the address stays, reads the voxels, can be shared
with another process as memory of cudaMalloc can, and may be asked for while a graph is
captured on another stream (also in the mode that forbids allocations) or on the context's."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _image(n=40, ctx=None):
    import sitk_b200 as sb
    a = np.random.default_rng(n).random((n, n + 1, n + 2), dtype=np.float32)
    return a, sb.DeviceImage.upload(a, ctx=ctx)


def _read(rt, ptr, like):
    out = np.empty_like(like)
    assert rt.cudaMemcpy(out.ctypes.data_as(ctypes.c_void_p), ctypes.c_void_p(ptr), ctypes.c_size_t(out.nbytes), 2) == 0
    return out


@pytest.mark.parametrize("made", ["upload", "smooth"])
def test_address(made):
    import torch
    torch.cuda.init()
    rt = ctypes.CDLL("libcudart.so.12")
    a, img = _image()
    if made == "smooth":
        img = img.smooth(1.0)
        a = img.to_host()
    at = img.device_ptr()
    assert at and img.device_ptr() == at
    np.testing.assert_array_equal(_read(rt, at, a), a)
    np.testing.assert_array_equal(img.to_host(), a)
    handle = (ctypes.c_char * 64)()
    assert rt.cudaIpcGetMemHandle(ctypes.byref(handle), ctypes.c_void_p(at)) == 0
    img.smooth(1.0).free()
    assert img.device_ptr() == at
    img.free()


@pytest.mark.parametrize("mode", [0, 1, 2])  # global, thread-local, relaxed
@pytest.mark.parametrize("own", [False, True])
def test_address_while_a_graph_is_captured(mode, own):
    import sitk_b200 as sb
    import torch
    rt = ctypes.CDLL("libcudart.so.12")
    ctx = sb.Context(0)
    a, img = _image(ctx=ctx)
    ctx.sync()
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    stream = ctypes.c_void_p(ctx.stream() if own else other.cuda_stream)
    assert rt.cudaStreamBeginCapture(stream, mode) == 0
    at = img.device_ptr()
    graph = ctypes.c_void_p()
    assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) == 0
    nodes = ctypes.c_size_t(7)
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(nodes)) == 0 and nodes.value == 0
    assert rt.cudaGraphDestroy(graph) == 0
    assert at and img.device_ptr() == at
    np.testing.assert_array_equal(_read(rt, at, a), a)
    img.free()
