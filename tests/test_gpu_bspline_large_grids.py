"""B-spline grids of many coefficients: on both sides of where they stop crossing in a pinned
copy, far more cells than samples, one metric over small and large grids in turn, and
coefficients that are not finite. Against the oracle (test_gpu_bspline_cells.py)."""
import numpy as np
import pytest

from test_gpu_bspline_cells import _case, _noise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(29, 29, 28), (29, 29, 29), (29, 29, 30), (60, 33, 40)])
@pytest.mark.parametrize("count", [900, None])
def test_both_sides_of_the_pinned_copy(oracle_lib, mesh, count):
    samples = None if count is None else np.random.default_rng(count).integers(0, 24 ** 3, count)
    _case(oracle_lib, 24, mesh, samples, _noise(0.5))


@pytest.mark.parametrize("bad", [np.nan, -np.inf, 1e300])
def test_coefficients_that_are_not_numbers(oracle_lib, bad):
    def coef(k):
        c = _noise(0.5)(k)
        c[k // 3 + 40] = bad
        return c
    _case(oracle_lib, 24, (30, 31, 30), None, coef)


def test_no_displacement(oracle_lib):
    _case(oracle_lib, 24, (30, 31, 30), None, np.zeros)


def test_grids_in_turn():
    import sitk_b200 as sb
    from conftest import small_pair
    from sitk_b200.transforms import BSplineTransform
    n = 24
    p = small_pair(n=n, seed=13, rot=6.0, trans=2.0)
    f, m = sb.DeviceImage.upload(p.fixed), sb.DeviceImage.upload(p.moving)
    ts = []
    for mesh in ((4, 4, 4), (31, 31, 31), (28, 28, 28), (40, 35, 33), (2, 2, 2)):
        t = BSplineTransform.from_image_domain(f.geo, mesh)
        t.set_parameters(0.5 * np.random.default_rng(sum(mesh)).standard_normal(t.nparams))
        ts.append(t)
    alone = [sb.DeviceMattesMetric.from_device(f, m, 32).evaluate(t) for t in ts]
    metric = sb.DeviceMattesMetric.from_device(f, m, 32)
    for k in [0, 1, 2, 3, 4, 3, 2, 1, 0, 3, 0]:
        r = metric.evaluate(ts[k])
        assert r.value == alone[k].value and r.valid_points == alone[k].valid_points
        assert metric.value(ts[k]) == r.value
        scale = np.max(np.abs(alone[k].derivative))
        assert np.max(np.abs(r.derivative - alone[k].derivative)) <= 1e-12 * scale  # (FP64 atomics: another order)
