"""A training step's gradients at batch sizes that leave tiles, K slices and column sums part
full, and below the size the network was made for, against the FP64 restatement that
rounds where the network's operands are BF16 (tests/test_initnet.py, its tolerance).
The biases keep every unit's input far from zero, half of the units on and half off:
otherwise a unit within FP32 rounding of zero may fall on either side of its ReLU, which
moves one sample's share (1/batch) of that unit's gradient."""
import numpy as np
import pytest

from test_initnet import _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,largest", [(1, 1), (3, 40), (17, 17), (40, 40)])
def test_gradients_at_batch(batch, largest):
    import torch
    from sitk_b200.initnet import InitNet
    rng = np.random.default_rng(batch)
    x = rng.standard_normal((batch, 32, 32, 32, 2)).astype(np.float32)
    t = rng.random((batch, 12)).astype(np.float32)
    net = InitNet(seed=5, max_batch=largest)
    state = net.state()
    for l in range(6):
        w = (state[l][0] * 0.05).astype(np.float32)
        b = np.where(np.arange(w.shape[0]) % 2 == 0, 2.0, -2.0).astype(np.float32)
        net.set(l, w, b)
        state[l] = (w, b)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    out, grads, loss = _reference(state, x, t)
    assert np.max(np.abs(net.forward(xd).cpu().numpy() - out)) <= 1e-2 * np.max(np.abs(out))
    assert abs(net.train_step(xd, td, lr=0.0) - loss) <= 1e-2 * loss
    first = [net.get(l, grads=True) for l in range(6)]
    for l in range(6):
        for got, ref in zip(first[l], grads[l]):
            assert np.max(np.abs(got - ref)) <= 1e-2 * np.max(np.abs(ref)), l
    net.train_step(xd, td, lr=0.0)  # repeated: the same bits
    for l in range(6):
        for a, b in zip(first[l], net.get(l, grads=True)):
            assert np.array_equal(a, b)
    net.close()
