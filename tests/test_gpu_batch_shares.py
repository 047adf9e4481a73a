"""A batch divides its pairs' samples and chunks evenly over the CTAs, across pairs and as
pairs stop. A pair's counts are integers, its chunks' sums are its own, so whatever else
is in the batch its result has the same bits as in a batch of its own: with pairs of
uneven sizes (sample counts on both sides of the chunks, shares and segments), with pairs
that stop at once beside pairs that go on, and with many more pairs than CTAs, where one
CTA finishes several pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _images(sizes):
    import sitk_b200 as sb
    from sitk_b200 import synth
    pairs = [synth.make_pair(n, 6, 70 + i, 4.0, 1.5, (0.97, 1.03)) for i, n in enumerate(sizes)]
    fixed = [sb.DeviceImage.upload(p.fixed) for p in pairs]
    # every third pair is an image and itself: it stops at its first evaluations
    moving = [sb.DeviceImage.upload(p.fixed if i % 3 == 1 else p.moving) for i, p in enumerate(pairs)]
    return fixed, moving


def _run(fixed, moving, sizes, seeds, bins, strategy, pct, iterations):
    from sitk_b200 import registration
    batch = registration.BatchRegistration(fixed, moving, bins=bins, kind=0, centers=[[(n - 1) / 2.0] * 3 for n in sizes],
                                           strategy=strategy, percentage=pct, seeds=seeds)
    start = np.tile(np.concatenate([np.eye(3).ravel(), np.zeros(3)]), (len(sizes), 1))
    params, results = batch.register(start, iterations=iterations, autotune=False)
    batch.close()
    return [(params[i].tobytes(), r.value, r.valid_points, r.iterations, r.stop_reason, r.evaluations)
            for i, r in enumerate(results)]


@pytest.mark.parametrize("sizes,copies,bins,strategy,pct,iterations", [
    ([16, 20, 33, 8, 41, 16, 25, 48], 1, 50, None, 1.0, 12),
    ([24, 47, 36, 52, 12], 1, 32, 2, 0.3, 12),
    ([64], 1, 100, None, 1.0, 5),
    ([8, 10, 9, 12, 11], 320, 32, 2, 0.5, 4)])
def test_a_pair_is_the_same_in_any_batch(sizes, copies, bins, strategy, pct, iterations):
    fixed, moving = _images(sizes)
    seeds = [5 + i for i in range(len(sizes))]
    alone = [_run([f], [m], [n], [s], bins, strategy, pct, iterations)[0]
             for f, m, n, s in zip(fixed, moving, sizes, seeds)]
    together = _run(fixed * copies, moving * copies, sizes * copies, seeds * copies, bins, strategy, pct, iterations)
    assert together == alone * copies
