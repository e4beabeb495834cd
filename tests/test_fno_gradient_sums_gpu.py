"""Sums of the surrogate's gradients over many pixels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,L,B", [(1, 1, 65536, 160), (3, 2, 262144, 32), (32, 32, 262144, 5)])
def test_long_sums_of_one_sign(rows, cols, L, B):
    """Constant gradients: every rounding of a chain has the same sign.  The bias sums
    are FP64 (one rounding of the result); a weight chain adds at most 256 products
    in FP32 (relative error below 256 roundings of 2^-24)."""
    from fastwigner_b200.fno import _Ops

    dY = torch.full((B, rows, L), 0.1, device="cuda")
    X = torch.full((B, cols, L), 0.7, device="cuda")
    out, bias = torch.empty(rows, cols, device="cuda"), torch.empty(rows, device="cuda")
    _Ops().wgrad_bias(rows, cols, L, dY, X, B, out, bias)
    y, x = float(dY[0, 0, 0]), float(X[0, 0, 0])
    assert ((bias.double() / (y * L * B)) - 1).abs().max() <= 2.0 ** -23
    assert ((out.double() / (y * x * L * B)) - 1).abs().max() <= 256 * 2.0 ** -24


def test_projection_bias_sums_add_in_fp64():
    """The hidden biases' gradients of a constant field: 65536 pixels give 16384 times
    what 4 do, up to the rounding of the two results."""
    from fastwigner_b200.fno import FNO2d

    net = FNO2d(seed=6)
    P = net.params
    res = []
    for L in (4, 65536):
        V, d = torch.full((1, 32, L), 0.3, device="cuda"), torch.full((1, L), 0.1, device="cuda")
        g = [torch.empty_like(P[k]) for k in ("Q1", "c1", "Q2", "c2")]
        net.ops.project_bwd(L, 1, V, P["Q1"], P["c1"], P["Q2"], d, torch.empty_like(V), *g)
        res.append(g)
    for i in (1, 3):
        a, b = res[0][i].double() * (65536 // 4), res[1][i].double()
        assert ((a - b).abs() <= 2.0 ** -23 * b.abs()).all()
