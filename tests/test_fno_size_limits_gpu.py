"""Networks and grids past the fused kernels' limits run on the general products."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_grid_of_more_columns_than_the_fused_layers_take():
    from fastwigner_b200.fno import FNO2d

    net = FNO2d(seed=1, layers=2)
    G0, G1 = 32, 65540
    X = np.random.default_rng(0).uniform(0, 1, (1, 3))
    xs, ps = np.linspace(-1, 1, G1, endpoint=False), np.linspace(-1, 1, G0, endpoint=False)
    a, b = net.forward(X, xs, ps, cache=False), net.forward(X, xs, ps, cache=True)
    assert (a - b).abs().max() <= 2e-5 * b.abs().max()
    net.backward(torch.ones_like(b))
    assert all(torch.isfinite(g).all() for g in net.grads.values())


@pytest.mark.parametrize("rows,cols", [(4100, 3), (1, 4100)])
def test_weight_gradients_wider_than_the_kernel_takes(rows, cols):
    from fastwigner_b200.fno import _Ops

    g = torch.Generator(device="cuda").manual_seed(rows)
    B, L = 2, 64
    dY, X = torch.randn(B, rows, L, device="cuda", generator=g), torch.randn(B, cols, L, device="cuda", generator=g)
    out, bias = torch.empty(rows, cols, device="cuda"), torch.empty(rows, device="cuda")
    _Ops().wgrad_bias(rows, cols, L, dY, X, B, out, bias)
    # sums of 128 products of unit variance at the tensor-core products' 1e-6 of a term
    assert (out.double() - torch.einsum("brl,bcl->rc", dY.double(), X.double())).abs().max() < 1e-6 * 128 ** 0.5 * 10
    assert (bias.double() - dY.double().sum(dim=(0, 2))).abs().max() < 1e-5
