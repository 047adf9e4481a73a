"""The initialiser on inputs, targets and outputs that start on an odd float of their buffer:
the bits of the same values in a buffer of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _view(t, first):
    import torch
    buf = torch.zeros(t.numel() + first, dtype=torch.float32, device="cuda")
    v = buf[first:].view(t.shape)
    v.copy_(t)
    return v


@pytest.mark.parametrize("first", [1, 2, 3])
@pytest.mark.parametrize("batch", [1, 3])
def test_views_that_start_on_any_float(batch, first):
    import torch
    from sitk_b200 import initnet
    g = torch.Generator().manual_seed(batch)
    x = torch.randn((batch, 32, 32, 32, 2), generator=g).cuda()
    t = torch.randn((batch, 12), generator=g).cuda()
    xv, tv = _view(x, first), _view(t, first)
    assert xv.data_ptr() % 16 == 4 * first
    whole, view = (initnet.InitNet(seed=3, max_batch=4) for _ in range(2))
    assert torch.equal(whole.forward(x), view.forward(xv))
    assert whole.train_step(x, t, 1e-3) == view.train_step(xv, tv, 1e-3)
    for l in range(initnet.N_LAYERS):
        for a, b in zip(whole.get(l) + whole.get(l, grads=True), view.get(l) + view.get(l, grads=True)):
            np.testing.assert_array_equal(a, b)
    out = torch.full((batch * 12 + 4,), -7.0, device="cuda")
    torch.cuda.synchronize()
    L = initnet._bind()
    assert L.mi_initnet_forward(view.handle, batch, xv.data_ptr(), out.data_ptr() + 4 * first) == 0
    assert torch.equal(out[first:first + 12 * batch].view(batch, 12), whole.forward(x))
    assert torch.all(out[:first] == -7.0) and torch.all(out[first + 12 * batch:] == -7.0)
