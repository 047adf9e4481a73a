"""Objects made and freed in one thread while another thread captures a graph on a stream of
its own: the capture ends well, and so do registrations of a batch (whose passes are captured).
Freeing an image whose address was given out waits for the work of every stream."""
import ctypes
import threading

import numpy as np
import pytest

from conftest import small_pair

pytestmark = pytest.mark.gpu


def _objects(lent):
    import sitk_b200 as sb
    p = small_pair(n=16, seed=5)
    ctx = sb.Context(0)
    f, m = sb.DeviceImage.upload(p.fixed, ctx=ctx), sb.DeviceImage.upload(p.moving, ctx=ctx)
    if lent:
        assert f.device_ptr() and m.device_ptr()
    sb.DeviceMattesMetric.from_device(f, m, 16).close()
    f.smooth(1.0).free()
    f.free()
    m.free()
    ctx.close()


@pytest.mark.parametrize("lent", [False, True])
def test_a_capture_in_another_thread_goes_on(lent):
    import torch
    _objects(lent)  # modules loaded
    rt = ctypes.CDLL("libcudart.so.12")
    stream = torch.cuda.Stream()
    at = ctypes.c_void_p(stream.cuda_stream)
    torch.cuda.synchronize()
    failed = []

    def work():
        try:
            _objects(lent)
        except Exception as e:
            failed.append(e)

    thread_local = 1
    assert rt.cudaStreamBeginCapture(at, thread_local) == 0
    th = threading.Thread(target=work)
    th.start()
    th.join()
    graph = ctypes.c_void_p()
    assert rt.cudaStreamEndCapture(at, ctypes.byref(graph)) == 0
    assert rt.cudaGraphDestroy(graph) == 0
    assert not failed


def test_batches_beside_frees():
    import sitk_b200 as sb
    from sitk_b200 import initnet
    from sitk_b200.registration import BatchRegistration
    stop, failed = threading.Event(), []

    def work():
        ctx = sb.Context(0)
        a = np.random.default_rng(1).random((8, 8, 8)).astype(np.float32)
        while not stop.is_set():
            try:
                sb.DeviceImage.upload(a, ctx=ctx).free()
            except Exception as e:
                failed.append(e)
                return

    ctx = sb.Context(0)
    pairs = [small_pair(n=24, seed=s) for s in range(3)]
    f = [sb.DeviceImage.upload(p.fixed, ctx=ctx) for p in pairs]
    m = [sb.DeviceImage.upload(p.moving, ctx=ctx) for p in pairs]
    th = threading.Thread(target=work)
    th.start()
    try:
        for k in range(60):  # a new graph for every number of iterations
            br = BatchRegistration(f, m, bins=16, kind=0, centers=[[11.5] * 3] * 3, strategy=2, percentage=0.3, seeds=[1, 2, 3])
            br.register(initnet.identity_params(3), iterations=5 + k, autotune=False)
            br.close()
    finally:
        stop.set()
        th.join()
    assert not failed


def test_a_lent_image_waits_for_every_stream():
    import sitk_b200 as sb
    import torch
    img = sb.DeviceImage.upload(np.zeros((8, 8, 8), np.float32))
    assert img.device_ptr()
    done, stream = torch.cuda.Event(), torch.cuda.Stream()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)  # about 50 ms
        done.record()
    img.free()
    assert done.query()
