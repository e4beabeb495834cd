"""The fused layer kernels of the FNO's inference path (fno_layer.cu) against
plain FP64 torch, stage by stage, at 1e-5 of each result's maximum (the bound
of the unfused tensor-core products): one and several x tiles, a ragged last
tile, fewer and more rows than the GPU has slots; then the whole fused forward
against the unfused one."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def swizzle(v):
    """[..., x, 32] <-> the kernels' pixel layout: 4-float piece q of pixel x at q ^ (x & 7)."""
    x = torch.arange(v.shape[-2], device=v.device)
    q = torch.arange(8, device=v.device)[None, :] ^ (x[:, None] & 7)
    idx = (4 * q[:, :, None] + torch.arange(4, device=v.device)).reshape(v.shape[-2], 32)
    return torch.gather(v, -1, idx.expand(v.shape))


def close(a, b, tol=1e-5):
    assert (a.double() - b).abs().max() <= tol * b.abs().max(), float((a.double() - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("B,G0,G1", [(1, 32, 128), (2, 48, 192), (3, 64, 36), (2, 256, 512), (1, 1024, 132)])
def test_layer_stages(B, G0, G1):
    from fastwigner_b200.fno import FNO2d

    net = FNO2d(seed=3)
    o, P = net.ops, net.params
    CS, Dpv, Dpiv, AA = net._grid(G0, G1)
    d = lambda t: t.double()  # noqa: E731
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    par, xs, ps = rnd(B, 3), rnd(G1), rnd(G0)
    v = torch.full((B, G0, G1, 32), float("nan"), device="cuda")
    fx = torch.full(((G1 + 127) // 128, B * G0, 32, 32), float("nan"), device="cuda")
    o.layer(0, B, G0, G1, P["W0"], P["b0"], CS=CS, NP=3, par=par, xs=xs, ps=ps, vout=v, fx=fx)
    feats = torch.cat([par[:, None, None, :].expand(B, G0, G1, 3), xs[None, None, :, None].expand(B, G0, G1, 1),
                       ps[None, :, None, None].expand(B, G0, G1, 1)], dim=3)
    v0 = d(feats) @ d(P["W0"]).T + d(P["b0"])
    close(swizzle(v), v0)
    close(fx.sum(0).view(B, G0, 32, 32), torch.einsum("bgxc,xk->bgck", v0, d(CS)))
    # p-transform, its inverse
    F2 = torch.empty((B, 32, 2, 512), device="cuda")
    o.pdft(B, G0, G1, fx, Dpv, F2)
    Fr = fx.double().sum(0).view(B, G0, 32, 2, 16).permute(0, 2, 1, 3, 4).reshape(B, 32, 2 * G0, 16)
    close(F2, (d(Dpv) @ Fr).reshape(B, 32, 2, 512))
    gx = torch.empty((B * G0, 32, 32), device="cuda")
    o.pidft(B, G0, F2, Dpiv, gx)
    Gr = (d(Dpiv) @ d(F2).reshape(B, 32, 64, 16)).reshape(B, 32, G0, 2, 16).permute(0, 2, 1, 3, 4).reshape(B, G0, 32, 32)
    close(swizzle(gx).view(B, G0, 32, 32), Gr)
    # a layer (in place) and the last layer with the projection
    vin = rnd(B, G0, G1, 32)
    pre = torch.einsum("bgck,kx->bgxc", Gr, d(AA)) + d(vin) @ d(P["W1"]).T + d(P["b1"])
    v = swizzle(vin).contiguous()
    out = torch.full((B, G0, G1), float("nan"), device="cuda")
    o.layer(2, B, G0, G1, P["W1"], P["b1"], vin=v, gx=gx, AA=AA, Q1=P["Q1"], c1=P["c1"], Q2=P["Q2"], c2=P["c2"], out=out)
    gelu = torch.nn.functional.gelu
    close(out, gelu(pre @ d(P["Q1"]).T + d(P["c1"])) @ d(P["Q2"])[0] + d(P["c2"]))
    o.layer(1, B, G0, G1, P["W1"], P["b1"], act=1, vin=v, gx=gx, AA=AA, CS=CS, vout=v, fx=fx)
    close(swizzle(v), gelu(pre))
    close(fx.sum(0).view(B, G0, 32, 32), torch.einsum("bgxc,xk->bgck", gelu(pre), d(CS)))
    st = ctypes.c_int(7)
    assert o.lib.fw_fno_status(ctypes.byref(st), 0) == 0 and st.value == 0


@pytest.mark.parametrize("G0,G1", [(64, 64), (192, 160), (512, 384)])
def test_fused_forward_matches_unfused(G0, G1):
    from fastwigner_b200.fno import FNO2d

    net = FNO2d(seed=1)
    X = np.random.default_rng(0).uniform(0, 1, (3, 3))
    xs, ps = np.linspace(-1, 1, G1, endpoint=False), np.linspace(-1, 1, G0, endpoint=False)
    assert net._fused_layers(G0, G1)
    a, b = net.forward(X, xs, ps, cache=False), net.forward(X, xs, ps, cache=True)
    assert (a - b).abs().max() <= 2e-5 * b.abs().max()


@pytest.mark.parametrize("rows,cols,L,B", [(32, 32, 65536, 2), (1, 128, 4100, 3), (128, 32, 1028, 1), (32, 5, 132, 4),
                                           (33, 40, 4, 2)])
def test_weight_and_bias_gradients(rows, cols, L, B):
    """fw_fno_wgrad_bias: tiles of 32 x 32 with ragged edges, pixel ranges that end
    inside a 128-pixel stage, one to many ranges per sample."""
    from fastwigner_b200.fno import _Ops

    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    dY = torch.randn(B, rows, L, device="cuda", generator=g)
    X = torch.randn(B, cols, L, device="cuda", generator=g)
    out, bias = torch.full((rows, cols), float("nan"), device="cuda"), torch.full((rows,), float("nan"), device="cuda")
    _Ops().wgrad_bias(rows, cols, L, dY, X, B, out, bias)
    # sums of B L products of unit variance: FP32 chains of a few hundred terms, FP64 above
    tol = 1e-6 * (B * L) ** 0.5 * 10
    assert (out.double() - torch.einsum("brl,bcl->rc", dY.double(), X.double())).abs().max() < tol
    assert (bias.double() - dY.double().sum(dim=(0, 2))).abs().max() < tol


@pytest.mark.parametrize("G0,G1,B", [(32, 36, 1), (48, 192, 2), (64, 132, 3)])
def test_training_gradients_match_autograd(G0, G1, B):
    """One loss_and_grad + backward on the fused path (layers' and projection
    backward, weight gradients) against FP64 autograd, 2e-5 of each gradient's
    maximum (a gradient is a chain of about ten products of 1e-6 each)."""
    from fastwigner_b200.fno import FNO2d

    net = FNO2d(seed=2)
    assert net._fused_layers(G0, G1)
    rng = np.random.default_rng(7)
    X = rng.uniform(0, 1, (B, 3))
    xs, ps = np.linspace(-1, 1, G1, endpoint=False), np.linspace(-1, 1, G0, endpoint=False)
    T = torch.tensor(rng.normal(size=(B, G0, G1)), dtype=torch.float32, device="cuda")
    loss, dY = net.loss_and_grad(X, xs, ps, T)
    grads = net.backward(dY)
    p = {k: v.double().detach().requires_grad_() for k, v in net.params.items()}
    f32 = lambda a: torch.tensor(np.asarray(a), dtype=torch.float32, device="cuda").double()  # noqa: E731
    feats = torch.cat([f32(X)[:, :, None, None].expand(B, 3, G0, G1), f32(xs)[None, None, None, :].expand(B, 1, G0, G1),
                       f32(ps)[None, None, :, None].expand(B, 1, G0, G1)], dim=1)
    ch = lambda W, b, u: torch.einsum("oi,bixy->boxy", W, u) + b[None, :, None, None]  # noqa: E731
    kp = np.concatenate([np.arange(16), np.arange(G0 - 16, G0)])
    v = ch(p["W0"], p["b0"], feats)
    for l in range(4):
        F = torch.fft.rfft2(v, norm="forward")[:, :, kp, :16].reshape(B, 32, 512)
        O = torch.einsum("bik,iok->bok", F, torch.complex(p[f"R{l}"][:, :, 0], p[f"R{l}"][:, :, 1])).reshape(B, 32, 32, 16)
        full = torch.zeros((B, 32, G0, G1 // 2 + 1), dtype=O.dtype, device="cuda")
        full[:, :, kp, :16] = O
        y = torch.fft.irfft(torch.fft.ifft(full, dim=2, norm="forward"), n=G1, dim=3, norm="forward")
        v = y + ch(p[f"W{l + 1}"], p[f"b{l + 1}"], v)
        if l < 3:
            v = torch.nn.functional.gelu(v)
    Y = ch(p["Q2"], p["c2"], torch.nn.functional.gelu(ch(p["Q1"], p["c1"], v)))[:, 0]
    ((Y - T.double()) ** 2).sum(dim=(1, 2)).div((T.double() ** 2).sum(dim=(1, 2))).mean().backward()
    for k, t in p.items():
        close(grads[k], t.grad, 2e-5)
