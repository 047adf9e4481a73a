"""Correlation of an overlap whose mean lies far, in its own standard deviations, from the rest
of the moving volume or of the fixed samples: as near the value in 64 bits (sums exact) as
where it does not, and the same derivative. One sample a thread and trees of 20 sums:
each of the three sums is off by at most 20·2^-53 of its terms, twice that with the shift's
cancellation; the value takes five of them, with |sfm| at most twice below its terms."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, IN = 48, 28
SHIFT = (0.3, 0.2, 0.4)
TOL = 2 * 2 * 5 * 20 * 2.0 ** -53


def _volumes(off, side):
    rng = np.random.default_rng(9)
    base = rng.standard_normal((N, N, N)).astype(np.float32)
    fixed = (base + 0.5 * rng.standard_normal((N, N, N))).astype(np.float32)
    moving = base.copy()
    outer = np.ones((N, N, N), bool)
    outer[:IN + 1, :IN + 1, :IN + 1] = False
    if side == "moving":
        moving[outer] += off
    else:
        fixed[outer] += off
    return fixed, moving


def _metric(fixed, moving, side):
    import sitk_b200 as sb
    z, y, x = (a.ravel() for a in np.meshgrid(*[np.arange(IN)] * 3, indexing="ij"))
    inner = x + N * (y + N * z)
    samples, mmask = inner, None
    if side == "fixed":  # the other samples see masked voxels only
        samples = np.concatenate([inner, np.flatnonzero(np.arange(N ** 3) // (N * N) >= IN + 2)])
        mmask = np.zeros((N, N, N), np.uint8)
        mmask[:IN + 1, :IN + 1, :IN + 1] = 1
    m = sb.DeviceCorrelationMetric.from_device_sampled(sb.DeviceImage.upload(fixed), sb.DeviceImage.upload(moving),
                                                       samples=samples, moving_mask=mmask)
    return m, (z, y, x)


@pytest.mark.parametrize("side", ["moving", "fixed"])
@pytest.mark.parametrize("off", [0.0, 0.7, 3.0, 30.0, 300.0, 3e4])
def test_value_and_derivative(side, off):
    import sitk_b200 as sb
    fixed, moving = _volumes(off, side)
    metric, (z, y, x) = _metric(fixed, moving, side)
    v = np.zeros(z.size)
    M = moving.astype(np.float64)
    for d in range(8):
        w = [SHIFT[a] if d >> a & 1 else 1 - SHIFT[a] for a in range(3)]
        v += w[0] * w[1] * w[2] * M[z + (d >> 2), y + (d >> 1 & 1), x + (d & 1)]
    f = fixed.astype(np.float64)[z, y, x]
    a, b = f - math.fsum(f) / f.size, v - math.fsum(v) / v.size
    sff, smm, sfm = math.fsum(a * a), math.fsum(b * b), math.fsum(a * b)
    want = -sfm * sfm / (sff * smm)
    t = sb.TranslationTransform(SHIFT)
    r = metric.evaluate(t)
    assert r.valid_points == z.size
    assert abs(r.value - want) <= TOL * abs(want) and abs(metric.value(t) - want) <= TOL * abs(want)
    plain, _ = _metric(*_volumes(0.0, side), side)
    d0 = plain.evaluate(t).derivative
    assert np.max(np.abs(r.derivative - d0)) <= 1e-12 * np.max(np.abs(d0))
