"""Objects freed after their context was destroyed, in every order, as a garbage collector may
finalise them; and what the context kept goes back to the device with the last of them."""
import itertools

import numpy as np
import pytest

from conftest import small_pair

pytestmark = pytest.mark.gpu


def _objects(sb, ctx):
    from sitk_b200 import initnet
    from sitk_b200.registration import BatchRegistration
    p = small_pair(n=20, seed=3)
    f, m = sb.DeviceImage.upload(p.fixed, ctx=ctx), sb.DeviceImage.upload(p.moving, ctx=ctx)
    metric = sb.DeviceMattesMetric.from_device_sampled(f, m, bins=16, strategy=2, percentage=0.5, seed=1)
    metric.evaluate(sb.TranslationTransform((0.1, 0.2, 0.3)))
    ncc = sb.DeviceCorrelationMetric.from_device(f, m)
    ncc.evaluate(sb.TranslationTransform((0.1, 0.2, 0.3)))
    br = BatchRegistration([f], [m], bins=16, kind=0, centers=[[9.5] * 3], strategy=2, percentage=0.5, seeds=[1])
    br.register(initnet.identity_params(1), iterations=3, autotune=False)
    net = initnet.InitNet(seed=1, max_batch=1, ctx=ctx)
    return [lambda: (f.free(), m.free()), metric.close, ncc.close, br.close, net.close]


@pytest.mark.parametrize("order", list(itertools.islice(itertools.permutations(range(5)), 0, 120, 17)))
def test_objects_may_outlive_their_context(order):
    import sitk_b200 as sb
    import torch
    torch.cuda.synchronize()
    before = None
    for turn in range(3):
        ctx = sb.Context(0)
        free = _objects(sb, ctx)
        first, rest = order[0], order[1:]
        free[first]()
        ctx.close()
        for k in rest:
            free[k]()
        torch.cuda.synchronize()
        now = torch.cuda.mem_get_info()[0]
        if turn:
            assert now >= before - (8 << 20), (turn, before, now)  # (the first turn loads modules)
        before = now


def test_an_image_is_whole_after_its_context():
    import sitk_b200 as sb
    a = np.random.default_rng(2).random((9, 8, 7)).astype(np.float32)
    ctx = sb.Context(0)
    img = sb.DeviceImage.upload(a, ctx=ctx)
    ctx.close()
    np.testing.assert_array_equal(img.to_host(), a)
    img.free()
