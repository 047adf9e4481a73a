"""Mean squares and correlation where their pass can go wrong: sample counts around a warp,
a CTA and the grid, volumes one or two voxels thick, BF16 and layered or 3-D textures, poses on
cell faces and past the volume's edge, a constant overlap, values far from the shift the
pass subtracts, and NaN. The oracle, within the reference's band (test_gpu_moments.py)."""
import numpy as np
import pytest

from conftest import small_pair

pytestmark = pytest.mark.gpu

BAND = 1e-9


def _rel(g, c):
    return np.abs(np.asarray(g) - np.asarray(c)) / (1.0 + np.abs(np.asarray(c)))


def _run(oracle, fixed, moving, t, which, samples=None, mmask=None, texture="auto"):
    import sitk_b200 as sb
    cls = sb.DeviceMeanSquaresMetric if which == "ms" else sb.DeviceCorrelationMetric
    f, m = sb.DeviceImage.upload(fixed), sb.DeviceImage.upload(moving)
    metric = cls.from_device_sampled(f, m, samples=samples, moving_mask=mmask, texture=texture)
    gf, gm = (oracle.make_geometry(v.shape[::-1]) for v in (fixed, moving))
    fn = oracle.mean_squares if which == "ms" else oracle.correlation
    ref = fn(fixed, gf, moving, gm, t.kind, t.params, t.fixed_params, draw=samples, mmask=mmask)
    r = metric.evaluate(t)
    v = metric.value(t)
    return r, v, ref


def _same(r, v, ref):
    assert r.valid_points == ref["valid"]
    assert _rel(r.value, ref["value"]) <= BAND and _rel(v, ref["value"]) <= BAND
    assert np.max(_rel(r.derivative, ref["derivative"])) <= BAND


@pytest.mark.parametrize("which", ["ms", "ncc"])
@pytest.mark.parametrize("count", [1, 2, 31, 33, 127, 129, 5000])
def test_sample_counts(oracle_lib, which, count):
    import sitk_b200 as sb
    p = small_pair(n=24, seed=2)
    t = sb.Euler3DTransform((0.03, -0.02, 0.05), (0.4, -0.3, 0.6), [11.5] * 3)
    samples = np.random.default_rng(count).integers(0, 24 ** 3, count)
    _same(*_run(oracle_lib, p.fixed, p.moving, t, which, samples=samples))


@pytest.mark.parametrize("which", ["ms", "ncc"])
@pytest.mark.parametrize("texture", ["auto", "3d"])
@pytest.mark.parametrize("shift", [(0.0, 0.0, 0.0), (1.0, 0.0, -2.0), (0.5, 0.5, 0.5), (7.25, -6.5, 0.0), (40.0, 0.0, 0.0)])
def test_faces_edges_and_no_overlap(oracle_lib, which, texture, shift):
    import sitk_b200 as sb
    p = small_pair(n=20, seed=4)
    _same(*_run(oracle_lib, p.fixed, p.moving, sb.TranslationTransform(shift), which, texture=texture))


@pytest.mark.parametrize("which", ["ms", "ncc"])
@pytest.mark.parametrize("shape", [(1, 9, 8), (2, 7, 33), (9, 1, 6), (5, 6, 1), (2, 2, 2)])
def test_thin_volumes(oracle_lib, which, shape):
    import sitk_b200 as sb
    rng = np.random.default_rng(sum(shape))
    fixed, moving = (rng.random(shape).astype(np.float32) * 100 for _ in range(2))
    t = sb.AffineTransform(np.eye(3) + 0.01, (0.2, -0.1, 0.15), (0.0, 0.0, 0.0))
    _same(*_run(oracle_lib, fixed, moving, t, which))


def test_correlation_far_from_its_shift(oracle_lib):
    """The samples see a small, nearly constant part of a moving volume whose mean is far
    away: the pass repeats with the means it found."""
    import sitk_b200 as sb
    rng = np.random.default_rng(9)
    moving = np.full((24, 24, 24), 1e4, dtype=np.float32)
    moving[:8, :8, :8] = 3.0 + 0.01 * rng.random((8, 8, 8))
    fixed = (50 + rng.random((24, 24, 24))).astype(np.float32)
    samples = np.array([x + 24 * (y + 24 * z) for z in range(6) for y in range(6) for x in range(6)])
    t = sb.TranslationTransform((0.3, 0.2, 0.4))
    _same(*_run(oracle_lib, fixed, moving, t, "ncc", samples=samples))


@pytest.mark.parametrize("value", [0.0, 7.0])
def test_correlation_of_a_constant_overlap_is_degenerate(oracle_lib, value):
    import sitk_b200 as sb
    moving = np.full((20, 20, 20), 123.25, dtype=np.float32)
    moving[:10] = value
    fixed = np.random.default_rng(1).random((20, 20, 20)).astype(np.float32)
    samples = np.arange(20 * 20 * 5)
    r, v, ref = _run(oracle_lib, fixed, moving, sb.TranslationTransform((0.0, 0.0, 0.5)), "ncc", samples=samples)
    assert ref["value"] == np.finfo(np.float64).max
    assert r.value == ref["value"] and v == ref["value"] and not np.any(r.derivative)


@pytest.mark.parametrize("which", ["ms", "ncc"])
def test_nan_reaches_the_value(which):
    import sitk_b200 as sb
    p = small_pair(n=20, seed=6)
    moving = p.moving.copy()
    moving[10, 10, 10] = np.nan
    cls = sb.DeviceMeanSquaresMetric if which == "ms" else sb.DeviceCorrelationMetric
    metric = cls.from_device(sb.DeviceImage.upload(p.fixed), sb.DeviceImage.upload(moving))
    t = sb.TranslationTransform((0.25, 0.25, 0.25))
    assert np.isnan(metric.value(t)) and np.isnan(metric.evaluate(t).value)
