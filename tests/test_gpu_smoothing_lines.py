"""The line kernels of the recursive Gaussian at the edges of their shapes: lines around
the chunks of 8 and 32 steps, the shortest ones, odd and even middles, line counts that
leave a warp's 16 lines part full, and lines past what shared memory holds; each set of
smoothed axes (the first pass widens, the last narrows). The oracle's bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(4, 5, 7), (7, 4, 6), (8, 9, 17), (31, 6, 5), (32, 33, 4), (65, 17, 9), (97, 35, 33),
                                  (1727, 4, 5), (1728, 5, 4), (5, 1814, 4), (4, 1815, 5),
                                  (5, 4, 1814), (4, 5, 1816)])
def test_lines_of_any_length_are_the_oracles(oracle_lib, size):
    import sitk_b200 as sb
    nx, ny, nz = size
    v = (np.random.default_rng(nx + ny + nz).standard_normal((nz, ny, nx)) * 100 + 50).astype(np.float32)
    sp = (1.0, 1.2, 0.9)
    g = oracle_lib.make_geometry(size, spacing=sp)
    img = sb.DeviceImage.upload(v, sp)
    for sigma in ((2.0, 1.5, 1.0), (3.0, 0.0, 0.0), (0.0, 3.0, 0.0), (0.0, 0.0, 3.0), (1.0, 0.0, 2.0), (0.0, 1.0, 1.0),
                  (0.0, 0.0, 0.0)):
        np.testing.assert_array_equal(img.smooth(sigma).to_host(), oracle_lib.recursive_gaussian(v, g, sigma))


@pytest.mark.parametrize("size", [(183, 228, 223), (185, 220, 227), (170, 231, 224)])
def test_many_long_lines_are_the_oracles(oracle_lib, size):
    # enough lines longer than 219 for the segment-wise form: last segments of 4, 7, 12, 15, 16 and
    # 19 elements, warps with lines missing, f32 and f64 on either side
    import sitk_b200 as sb
    nx, ny, nz = size
    v = (np.random.default_rng(nx + ny + nz).standard_normal((nz, ny, nx)) * 100 + 50).astype(np.float32)
    sp = (1.0, 1.2, 0.9)
    g = oracle_lib.make_geometry(size, spacing=sp)
    img = sb.DeviceImage.upload(v, sp)
    for sigma in ((2.0, 1.5, 1.0), (0.0, 3.0, 0.0), (0.0, 1.0, 4.0)):
        np.testing.assert_array_equal(img.smooth(sigma).to_host(), oracle_lib.recursive_gaussian(v, g, sigma))
