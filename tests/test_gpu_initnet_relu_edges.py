"""The initialiser's ReLU at the edge of zero: a unit whose FP32 input is positive but below
BF16's least value still passes its gradient back; one at zero, at minus zero or below does
not. Each layer's units are all set to one input by its bias."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layer", range(5))
@pytest.mark.parametrize("z,passes", [(1e-45, True), (4e-41, True), (1e-38, True), (0.5, True), (0.0, False), (-0.0, False),
                                      (-1e-45, False), (-0.5, False), (np.nan, False)])
def test_gradient_passes_where_the_input_is_positive(layer, z, passes):
    import torch
    from sitk_b200 import initnet
    net = initnet.InitNet(seed=1, max_batch=2)
    state = net.state()
    for l, (w, b) in enumerate(state):
        if l == layer:
            w, b = np.zeros_like(w), np.full_like(b, z)
        elif l < layer:
            w, b = np.zeros_like(w), np.ones_like(b)
        else:  # every unit above is positive, and passes a positive gradient down
            w, b = np.full_like(w, 2.0 ** -6), np.ones_like(b)
        net.set(l, w, b)
    g = torch.Generator().manual_seed(1)
    x = torch.randn((2, 32, 32, 32, 2), generator=g).cuda()
    net.train_step(x, torch.full((2, 12), -50.0, device="cuda"), 0.0)
    gb = net.get(layer, grads=True)[1]
    if passes:
        assert np.all(np.isfinite(gb)) and np.all(gb > 0)
    else:
        assert np.all(gb == 0)


def test_no_output_of_a_dead_layer():
    import torch
    from sitk_b200 import initnet
    net = initnet.InitNet(seed=2, max_batch=1)
    w, b = net.get(4)
    net.set(4, np.zeros_like(w), np.full_like(b, -1.0))
    w, b = net.get(5)
    net.set(5, w, np.zeros_like(b))
    y = net.forward(torch.ones((1, 32, 32, 32, 2), device="cuda"))
    assert torch.all(y == 0)
