"""Loss gradients at any address."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("net_kw,G0,G1", [(dict(), 32, 36), (dict(), 34, 34), (dict(width=16), 32, 64)])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_backward_takes_a_loss_gradient_at_any_address(net_kw, G0, G1, off):
    from fastwigner_b200.fno import FNO2d

    net = FNO2d(seed=2, **net_kw)
    B = 2
    rng = np.random.default_rng(1)
    X = rng.uniform(0, 1, (B, 3))
    xs, ps = np.linspace(-1, 1, G1, endpoint=False), np.linspace(-1, 1, G0, endpoint=False)
    d = torch.tensor(rng.normal(size=(B, G0, G1)), dtype=torch.float32, device="cuda")
    buf = torch.empty(d.numel() + 4, device="cuda")
    view = buf[off:off + d.numel()].view(d.shape)
    view.copy_(d)
    assert view.is_contiguous() and view.data_ptr() % 16 == 4 * off
    net.forward(X, xs, ps)
    want = {k: g.clone() for k, g in net.backward(d).items()}
    net.forward(X, xs, ps)
    got = net.backward(view)
    for k in want:
        assert torch.equal(got[k], want[k]), k
