"""The B-spline pass in cell order where it can go wrong: more cells than samples, one cell,
samples outside the grid's valid region, duplicate and few samples, no displacement (every
point on a voxel: the exact chain), displacements past the volume, coefficients that are
not finite. Decisions, value and derivative against the oracle (test_gpu_bspline.py)."""
import numpy as np
import pytest

from conftest import small_pair
from test_gpu_bspline import _records

pytestmark = pytest.mark.gpu


def _case(oracle, n, mesh, samples, coef, domain=1.0, bins=32):
    import sitk_b200 as sb
    from sitk_b200.transforms import BSplineTransform
    p = small_pair(n=n, seed=13, rot=6.0, trans=2.0)
    f, m = sb.DeviceImage.upload(p.fixed), sb.DeviceImage.upload(p.moving)
    metric = sb.DeviceMattesMetric.from_device_sampled(f, m, samples=samples, bins=bins)
    t = BSplineTransform((0.0, 0.0, 0.0), (domain * n,) * 3, np.eye(3), mesh)
    t.set_parameters(coef(t.nparams))
    g = oracle.make_geometry((n, n, n))
    draw = np.arange(n ** 3) if samples is None else np.asarray(samples)
    ref = oracle.bspline_mattes(p.fixed, g, p.moving, g, bins, t.fixed_params, t.params, draw=draw, per_sample=True)
    dev = metric.sample_order().astype(np.int64)
    o_ord, d_ord = np.argsort(draw, kind="stable"), np.argsort(dev, kind="stable")
    order = np.empty_like(o_ord)
    order[d_ord] = o_ord
    rec, st = _records(metric, t), ref["status"][order]
    np.testing.assert_array_equal(rec != 0, st == 2)
    ok = st == 2
    np.testing.assert_array_equal(rec[ok] & 0xff, ref["mi"][order][ok])
    np.testing.assert_array_equal(rec[ok] >> 8, ref["fi"][order][ok])
    mv = metric.evaluate(t)
    assert mv.valid_points == ref["valid"]
    if ref["valid"] and np.isfinite(ref["value"]):
        assert abs(mv.value - ref["value"]) <= 1e-5 * abs(ref["value"])
        scale = np.max(np.abs(ref["derivative"]))
        assert np.max(np.abs(mv.derivative - ref["derivative"])) <= 1e-4 * scale
    assert metric.value(t) == mv.value
    return mv


def _noise(amp, seed=1):
    return lambda k: amp * np.random.default_rng(seed).standard_normal(k)


@pytest.mark.parametrize("mesh", [(1, 1, 1), (9, 7, 11), (2, 13, 1)])
@pytest.mark.parametrize("count", [40, 3000])
def test_meshes_and_sample_counts(oracle_lib, mesh, count):
    samples = np.random.default_rng(count).integers(0, 24 ** 3, count)
    _case(oracle_lib, 24, mesh, samples, _noise(0.7))


@pytest.mark.parametrize("bins", [8, 50, 128])
def test_bins(oracle_lib, bins):
    _case(oracle_lib, 24, (3, 4, 2), None, _noise(0.7), bins=bins)


def test_grid_smaller_than_the_image(oracle_lib):
    _case(oracle_lib, 28, (3, 3, 3), None, _noise(0.6), domain=0.55)


def test_no_displacement(oracle_lib):
    _case(oracle_lib, 24, (3, 3, 3), None, np.zeros)


def test_whole_voxels(oracle_lib):
    _case(oracle_lib, 24, (3, 3, 3), None, np.ones)


def test_displacement_past_the_volume(oracle_lib):
    assert _case(oracle_lib, 24, (3, 3, 3), None, lambda k: np.full(k, 200.0)).valid_points == 0
    _case(oracle_lib, 24, (3, 3, 3), None, _noise(30.0))


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e300])
def test_coefficients_that_are_not_numbers(oracle_lib, bad):
    def coef(k):
        c = _noise(0.5)(k)
        c[k // 2] = bad
        return c
    _case(oracle_lib, 24, (4, 4, 4), None, coef)
