"""The walk order of a sample list: 8³ bricks (bricks of 2^bl voxels for the Mattes metric),
the order of the layout's keys, from keys of 32 bits and, where the bricks of a thin grid
pad past them, of 64; duplicates kept, masked samples dropped, NaN left out of the ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _key(flat, size, bl):
    flat = flat.astype(np.int64)
    x, y, z = flat % size[0], flat // size[0] % size[1], flat // (size[0] * size[1])
    nbx, nby = (size[0] + (1 << bl) - 1) >> bl, (size[1] + (1 << bl) - 1) >> bl
    brick = ((z >> bl) * nby + (y >> bl)) * nbx + (x >> bl)
    sb, m = bl - 3, (1 << (bl - 3)) - 1
    sub = (((z >> 3) & m) << sb | ((y >> 3) & m)) << sb | ((x >> 3) & m)
    return brick << (3 * bl) | sub << 9 | (z & 7) << 6 | (y & 7) << 3 | (x & 7)


@pytest.mark.parametrize("count,bl", [(300, 6), (9000, 4), (120, 6)])
def test_mattes_order(count, bl):
    import sitk_b200 as sb
    size = (37, 70, 45)
    rng = np.random.default_rng(count)
    v = rng.random(size[::-1]).astype(np.float32)
    v[3, 4, 5] = np.nan
    samples = rng.integers(0, v.size, count)
    mask = (rng.random(v.shape) > 0.25).astype(np.float32)
    img = sb.DeviceImage.upload(v)
    for m in (None, mask):
        metric = sb.DeviceMattesMetric.from_device_sampled(img, img, fixed_mask=m, samples=samples, bins=16)
        kept = samples if m is None else samples[mask.ravel()[samples] != 0]
        order = metric.sample_order()
        want = kept[np.argsort(_key(kept, size, bl), kind="stable")]
        np.testing.assert_array_equal(order, want)
        info = metric.info()
        f = v.ravel()[kept]
        assert info["fixed_min"] == np.nanmin(f) and info["fixed_max"] == np.nanmax(f)
        assert info["moving_min"] == np.nanmin(v) and info["moving_max"] == np.nanmax(v)


@pytest.mark.parametrize("size", [(40, 33, 21), (1, 1 << 27, 1)])
def test_mean_squares_order(size):
    import torch
    import sitk_b200 as sb
    rng = np.random.default_rng(1)
    n = size[0] * size[1] * size[2]
    v = torch.zeros(n, device="cuda")
    torch.cuda.synchronize()
    img = sb.DeviceImage.from_device_ptr(v.data_ptr(), size)
    samples = rng.integers(0, n, 5000)
    samples[::7] = samples[0]
    order = sb.DeviceMeanSquaresMetric.from_device_sampled(img, img, samples=samples).sample_order()
    np.testing.assert_array_equal(order, samples[np.argsort(_key(samples, size, 3), kind="stable")])
