"""Odd numbers of histogram bins, whose squares leave the tables of 32-bit words at odd places:
every launch form of the Mattes metric against the oracle (test_gpu_parity.py's contract), a
batch against its pairs by themselves, and a B-spline."""
import numpy as np
import pytest

from conftest import small_pair
from test_gpu_bspline_cells import _case, _noise
from test_gpu_parity import _compare

pytestmark = pytest.mark.gpu

ODD = [7, 9, 31, 33, 49, 63, 127]


@pytest.mark.parametrize("bins", ODD)
@pytest.mark.parametrize("kw", [dict(), dict(strategy=2, pct=0.3, seed=4), dict(moving_storage="bf16")],
                         ids=["all", "random", "bf16"])
def test_metric(oracle_lib, bins, kw):
    import sitk_b200 as sb
    n = 24
    p = small_pair(n=n, seed=5)
    t = sb.Euler3DTransform((0.02, -0.03, 0.01), (0.5, -0.25, 0.75), [11.5] * 3)
    _compare(oracle_lib, p, n, t, bins, **kw)


def test_the_fewest_bins(oracle_lib):
    """Five bins are one of intensities and four of padding: the information is zero, to the
    histogram's unit of 2^-22 a tap (four of them, so 2^-20 of the value's order of one)."""
    import sitk_b200 as sb
    n = 24
    p = small_pair(n=n, seed=5)
    t = sb.Euler3DTransform((0.02, -0.03, 0.01), (0.5, -0.25, 0.75), [11.5] * 3)
    metric = sb.DeviceMattesMetric.from_device(sb.DeviceImage.upload(p.fixed), sb.DeviceImage.upload(p.moving), 5)
    g = oracle_lib.make_geometry((n, n, n))
    ref = oracle_lib.evaluate(p.fixed, g, p.moving, g, 5, t.kind, t.params, t.fixed_params)
    r = metric.evaluate(t)
    assert r.valid_points == ref["valid"] and abs(ref["value"]) < 1e-12
    assert abs(r.value) <= 2.0 ** -20 and metric.value(t) == r.value


@pytest.mark.parametrize("bins", ODD)
def test_staged_tiles(bins):
    import sitk_b200 as sb
    from sitk_b200.metric import get_tile_staging, set_tile_staging
    p = small_pair(n=32, seed=5)
    metric = sb.DeviceMattesMetric.from_device(sb.DeviceImage.upload(p.fixed), sb.DeviceImage.upload(p.moving), bins)
    t = sb.Euler3DTransform((0.02, -0.03, 0.01), (0.5, -0.25, 0.75), [15.5] * 3)
    plain = metric.evaluate(t)
    set_tile_staging(metric, True)
    tiled = metric.evaluate(t)
    assert plain.value == tiled.value and plain.valid_points == tiled.valid_points
    scale = np.max(np.abs(plain.derivative))
    assert np.max(np.abs(plain.derivative - tiled.derivative)) <= 1e-4 * scale
    assert metric.value(t) == plain.value


@pytest.mark.parametrize("bins", ODD)
def test_batch(bins):
    import sitk_b200 as sb
    from sitk_b200 import registration
    sizes = [24, 33, 28]
    pairs = [small_pair(n=n, seed=30 + n, rot=5.0, trans=2.0) for n in sizes]
    fixed = [sb.DeviceImage.upload(p.fixed) for p in pairs]
    moving = [sb.DeviceImage.upload(p.moving) for p in pairs]
    centers = [[(n - 1) / 2.0] * 3 for n in sizes]
    batch = registration.BatchRegistration(fixed, moving, bins=bins, kind=0, centers=centers)
    start = np.tile(np.concatenate([np.eye(3).ravel(), np.zeros(3)]), (3, 1))
    _, results = batch.register(start, iterations=1, autotune=False)
    batch.close()
    for k, (f, m) in enumerate(zip(fixed, moving)):
        t = sb.AffineTransform(np.eye(3), (0.0, 0.0, 0.0), centers[k])
        r = registration.register_rsgd(sb.DeviceMattesMetric.from_device(f, m, bins), t, iterations=1)
        assert results[k].iterations == r.iterations and results[k].evaluations == r.evaluations
        assert abs(results[k].value - r.value) <= 1e-3 * abs(r.value)
        assert abs(results[k].valid_points - r.valid_points) <= max(2, 1e-4 * r.valid_points)


@pytest.mark.parametrize("bins", ODD)
def test_bspline(oracle_lib, bins):
    _case(oracle_lib, 24, (3, 4, 2), None, _noise(0.7), bins=bins)
