"""What objects hand on to the next one of a context (device blocks, pinned blocks,
texture arrays) carries nothing over: an object built from reused parts gives the bits
of one built in a fresh context, also with several contexts in several threads, and a
context can be destroyed and made again."""
import threading

import numpy as np
import pytest

from conftest import small_pair

pytestmark = pytest.mark.gpu

SHAPES = [(24, "f32", "auto", "mattes"), (24, "bf16", "auto", "mattes"), (24, "f32", "3d", "mattes"),
          (31, "f32", "auto", "ms"), (24, "f32", "auto", "ncc"), (31, "f32", "auto", "mattes")]


def _one(ctx, n, storage, texture, kind, seed):
    import sitk_b200 as sb
    p = small_pair(n=n, seed=seed)
    f, m = sb.DeviceImage.upload(p.fixed, ctx=ctx), sb.DeviceImage.upload(p.moving, ctx=ctx)
    cls = {"mattes": sb.DeviceMattesMetric, "ms": sb.DeviceMeanSquaresMetric, "ncc": sb.DeviceCorrelationMetric}[kind]
    metric = cls.from_device_sampled(f, m, strategy=sb.SAMPLING_RANDOM, percentage=0.5, seed=seed,
                                     moving_storage=storage, texture=texture)
    r = metric.evaluate(sb.Euler3DTransform((0.02, -0.03, 0.01), (0.5, -0.25, 0.75), [n / 2.0] * 3))
    s = f.smooth((1.0, 0.0, 2.0)).to_host()
    metric.close()
    f.free()
    m.free()
    return r.value, r.valid_points, r.derivative.tobytes(), s.tobytes()


def _fresh(shape, seed):
    import sitk_b200 as sb
    ctx = sb.Context(0)
    r = _one(ctx, *shape, seed)
    ctx.close()
    return r


def test_reused_parts_give_a_fresh_contexts_bits():
    import sitk_b200 as sb
    want = {(s, seed): _fresh(s, seed) for s in SHAPES for seed in (3, 4)}
    got = {}

    def work(name):
        ctx = sb.Context(0)
        for _ in range(3):
            for k in want:
                got.setdefault((name, k), []).append(_one(ctx, *k[0], k[1]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 3 * len(want)
    for (_, k), results in got.items():
        assert len(results) == 3 and all(r == want[k] for r in results), k
