"""B-spline derivative where support weights are exactly zero: every sample on the cells' lower
faces, so that the last control point of each of its axes has weight zero there. Those
coefficients' derivatives are exactly zero, as the sums of zeros they are; and where a weight
is subnormal, or the products of three are, the derivative is the oracle's."""
import numpy as np
import pytest

from conftest import small_pair

pytestmark = pytest.mark.gpu


def _evaluate(n, t):
    import sitk_b200 as sb
    p = small_pair(n=n, seed=13, rot=6.0, trans=2.0)
    f, m = sb.DeviceImage.upload(p.fixed), sb.DeviceImage.upload(p.moving)
    return p, sb.DeviceMattesMetric.from_device(f, m, 32).evaluate(t)


@pytest.mark.parametrize("mesh", [(20, 20, 20), (10, 10, 10), (20, 4, 5)])
def test_zero_weights_give_zero(mesh):
    from sitk_b200.transforms import BSplineTransform
    n = 20
    t = BSplineTransform((0.0, 0.0, 0.0), (float(n),) * 3, np.eye(3), mesh)
    t.set_parameters(0.3 * np.random.default_rng(1).standard_normal(t.nparams))
    _, r = _evaluate(n, t)
    assert r.valid_points > 0 and np.any(r.derivative)
    d = r.derivative.reshape(3, *reversed(t.grid_size))
    # A grid spacing of one voxel puts every sample on its cell's lower faces, where the fourth
    # control point of the cell has weight zero; the last plane of control points is no
    # other cell's.
    for axis, (m, plane) in enumerate(zip(mesh, (d[:, :, :, -1], d[:, :, -1], d[:, -1]))):
        if m == n:
            assert np.all(plane == 0.0), axis


@pytest.mark.parametrize("eps", [1e-13, 1e-14, 3e-13])
def test_subnormal_weights(oracle_lib, eps):
    from sitk_b200.transforms import BSplineTransform
    n = 16
    # the samples lie eps of a cell above the faces: weights of eps³/6 and products below FP32's range
    t = BSplineTransform((-eps, -eps, -eps), (float(n),) * 3, np.eye(3), (n, n, n))
    t.set_parameters(0.3 * np.random.default_rng(1).standard_normal(t.nparams))
    p, r = _evaluate(n, t)
    g = oracle_lib.make_geometry((n, n, n))
    ref = oracle_lib.bspline_mattes(p.fixed, g, p.moving, g, 32, t.fixed_params, t.params, draw=np.arange(n ** 3))
    assert r.valid_points == ref["valid"]
    d, want = (np.reshape(v, (3, n + 3, n + 3, n + 3))[:, -1, -1, -1] for v in (r.derivative, ref["derivative"]))
    # one cell's last control point: three weights of about eps³/6, far below FP32
    assert np.all(np.abs(d) <= 1e-30) and np.all(np.abs(want) <= 1e-30)
    scale = np.max(np.abs(ref["derivative"]))
    assert np.max(np.abs(r.derivative - ref["derivative"])) <= 1e-4 * scale
