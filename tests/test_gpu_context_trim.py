"""A trimmed context gives its spare device memory back to others, and its objects, and those
made after it, are unaffected; also while another thread works in a context of its own."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _work(sb, ctx, n=160):
    rng = np.random.default_rng(3)
    v = rng.random((n, n, n), dtype=np.float32)
    f, m = sb.DeviceImage.upload(v, ctx=ctx), sb.DeviceImage.upload(v[::-1].copy(), ctx=ctx)
    metric = sb.DeviceMattesMetric.from_device_sampled(f, m, bins=32, strategy=2, percentage=0.1, seed=1)
    s = f.smooth(1.5)
    r = metric.evaluate(sb.TranslationTransform((0.5, 0.25, -1.0)))
    out = (r.value, r.derivative.tobytes(), s.to_host().tobytes())
    for o in (s, f, m):
        o.free()
    return out, metric


def test_trim():
    import sitk_b200 as sb
    import torch
    ctx = sb.Context(0)
    want, metric = _work(sb, ctx)
    metric.close()
    torch.cuda.synchronize()
    kept = torch.cuda.mem_get_info()[0]
    ctx.trim()
    # (two images, FP64 volumes, texture array: over 80 MB at 160³)
    assert torch.cuda.mem_get_info()[0] - kept >= 60 << 20
    got, metric = _work(sb, ctx)
    assert got == want
    t = sb.TranslationTransform((0.5, 0.25, -1.0))
    before = metric.evaluate(t)
    ctx.trim()
    after = metric.evaluate(t)
    assert before.value == after.value == want[0]
    assert before.derivative.tobytes() == after.derivative.tobytes() == want[1]


def test_trim_beside_another_threads_context():
    import sitk_b200 as sb
    stop, failed, results = threading.Event(), [], set()

    def work():
        try:
            ctx = sb.Context(0)
            while not stop.is_set():
                out, metric = _work(sb, ctx, 48)
                metric.close()
                results.add(out)
        except Exception as e:
            failed.append(e)

    th = threading.Thread(target=work)
    th.start()
    try:
        ctx = sb.Context(0)
        for _ in range(30):
            out, metric = _work(sb, ctx, 48)
            metric.close()
            ctx.trim()
            results.add(out)
    finally:
        stop.set()
        th.join()
    assert not failed and len(results) == 1
