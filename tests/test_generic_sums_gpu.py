"""Observable sums of the generic passes' fused FP32 mid-point: the squares, the
weights and the sums are held in FP64 whatever the state's precision, as by sums
over the real-space values."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(P, X, W0, wx, wp, steps, per_instance=False):
    """`steps` steps of W' = W (all phases zero) through the C ABI: obs (steps, batch, M)."""
    import torch

    from fastwigner_b200 import _lib

    lib = _lib.load()
    B = W0.shape[0]
    W = torch.tensor(W0, dtype=torch.float32, device="cuda")
    one = lambda *s: torch.tensor([1.0, 0.0], device="cuda").expand(*s, 2).contiguous()  # noqa: E731
    tabV, tabK = one(P // 2 + 1, X), one(P, X // 2 + 1)
    wx, wp = (torch.tensor(w, dtype=torch.float64, device="cuda") for w in (wx, wp))
    M = 2 + wx.shape[-2] + wp.shape[-2]
    obs = torch.full((steps, B, M), float("nan"), dtype=torch.float64, device="cuda")
    d = _lib.WignerDesc()
    d.W, d.w_bstride, d.step_kind = W.data_ptr(), P * X, _lib.FW_STEP_FUSED
    d.tabV, d.tabK = tabV.data_ptr(), tabK.data_ptr()
    d.Mx, d.Mp, d.wx, d.wp = wx.shape[-2], wp.shape[-2], wx.data_ptr(), wp.data_ptr()
    if per_instance:
        d.wp_bstride = wp.shape[-2] * P
    d.obs_out, d.dxdp, d.in_scale = obs.data_ptr(), 1.0, 1.0
    plan = _lib.c_vp()
    _lib.check(lib.fw_wigner_plan_create(P, X, B, _lib.FW_F32, ctypes.byref(plan)))
    try:
        st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(lib.fw_wigner_propagate(plan, ctypes.byref(d), steps, st))
        torch.cuda.synchronize()
    finally:
        lib.fw_wigner_plan_destroy(plan)
    return obs.cpu().numpy()


@pytest.mark.parametrize("scale", [1e24, 1e-24])
@pytest.mark.parametrize("P,X", [(96, 100), (90, 14), (512, 24)])
def test_squares_of_a_state_of_any_scale(P, X, scale):
    rng = np.random.default_rng(P)
    W0 = np.abs(rng.normal(size=(2, P, X))).astype(np.float32).astype(np.float64) * scale
    W0 = W0.astype(np.float32)
    obs = _run(P, X, W0, np.ones((1, X)), np.ones((1, P)), 2)
    W = W0.astype(np.float64)
    # FP32 transforms of the state: a few roundings of 6e-8 each
    np.testing.assert_allclose(obs[0, :, 1], (W * W).sum(axis=(1, 2)), rtol=2e-6)
    np.testing.assert_allclose(obs[0, :, 0], W.sum(axis=(1, 2)), rtol=2e-6)


@pytest.mark.parametrize("per_instance", [False, True])
@pytest.mark.parametrize("P,X,Mp", [(96, 12, 1), (96, 12, 4), (12, 96, 2), (512, 24, 3), (1152, 36, 4)])
def test_weights_far_from_the_state(P, X, Mp, per_instance):
    """W = c at one point: sizes of radices 2, 3 and 4 transform it exactly (equal inputs
    give exact zeros), so every p-sum is w(p0) times the sum of W, whatever the
    weights elsewhere; FP64 leaves 1e-12 of their maximum (FP32 spectra: 1e-7)."""
    rng = np.random.default_rng(P + Mp)
    B = 3
    W0 = np.zeros((B, P, X), dtype=np.float32)
    W0[:, 0, 0] = [1.0, 3.0, 0.25]
    wp = rng.uniform(0, 1e4, size=(B if per_instance else 1, Mp, P))
    wp[..., 0] = rng.uniform(0, 1, size=wp.shape[:-1])
    obs = _run(P, X, W0, np.ones((2, X)), wp if per_instance else wp[0], 3, per_instance)
    w0 = np.broadcast_to(wp[..., 0], (B, Mp))
    for k in range(3):
        S = obs[k, :, :1]
        assert np.abs(obs[k, :, 4:] - w0 * S).max() <= 1e-12 * 1e4 * S.max()
        np.testing.assert_allclose(obs[k, :, 2:4], np.repeat(S, 2, axis=1), rtol=1e-12)
