"""Mean squares and correlation over moving volumes with infinite voxels, off and on the cell
faces, at every corner of a cell: the value is the infinity or the NaN that the reference's
weighted sum of the corners gives (the oracle)."""
import numpy as np
import pytest

from conftest import small_pair

pytestmark = pytest.mark.gpu


def _kind(v):
    return "nan" if np.isnan(v) else ("inf" if v == np.inf else ("-inf" if v == -np.inf else "finite"))


@pytest.mark.parametrize("which", ["ms", "ncc"])
@pytest.mark.parametrize("bad", [np.inf, -np.inf])
@pytest.mark.parametrize("corner", range(8))
@pytest.mark.parametrize("shift", [(0.25, 0.375, 0.5), (0.0, 0.25, 0.0), (1.0, -2.0, 0.0)])
def test_one_infinite_corner(oracle_lib, which, bad, corner, shift):
    import sitk_b200 as sb
    n = 12
    p = small_pair(n=n, seed=6)
    moving = p.moving.copy()
    # the samples fall into one cell, whose corner `corner` is infinite
    moving[5 + (corner >> 2), 5 + (corner >> 1 & 1), 5 + (corner & 1)] = bad
    at = [5 - int(np.floor(s)) for s in shift]
    samples = np.array([at[0] + n * (at[1] + n * at[2])] * 3 + [0])
    t = sb.TranslationTransform(shift)
    cls = sb.DeviceMeanSquaresMetric if which == "ms" else sb.DeviceCorrelationMetric
    metric = cls.from_device_sampled(sb.DeviceImage.upload(p.fixed), sb.DeviceImage.upload(moving), samples=samples)
    g = oracle_lib.make_geometry((n, n, n))
    fn = oracle_lib.mean_squares if which == "ms" else oracle_lib.correlation
    ref = fn(p.fixed, g, moving, g, t.kind, t.params, t.fixed_params, draw=samples)
    r = metric.evaluate(t)
    assert r.valid_points == ref["valid"]
    assert _kind(r.value) == _kind(metric.value(t)) == _kind(ref["value"])
    assert [_kind(d) for d in r.derivative] == [_kind(d) for d in ref["derivative"]]


def test_an_infinite_voxel_of_a_whole_volume():
    import sitk_b200 as sb
    p = small_pair(n=20, seed=6)
    moving = p.moving.copy()
    moving[10, 10, 10] = np.inf
    metric = sb.DeviceMeanSquaresMetric.from_device(sb.DeviceImage.upload(p.fixed), sb.DeviceImage.upload(moving))
    t = sb.TranslationTransform((0.25, 0.25, 0.25))
    assert metric.value(t) == np.inf and metric.evaluate(t).value == np.inf
