"""Plans of different lengths propagated by several threads at once: a launch's
shared-memory limit is not another thread's."""
import ctypes
import threading

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_lengths_from_several_threads(precision):
    import torch

    from fastwigner_b200 import _lib

    lib = _lib.load()
    rt = torch.float64 if precision == "float64" else torch.float32
    code = _lib.FW_F64 if precision == "float64" else _lib.FW_F32
    errors = []

    def work(P):
        try:
            X, M = 128, 4
            one = lambda *s: torch.tensor([1.0, 0.0], dtype=rt, device="cuda").expand(*s, 2).contiguous()  # noqa: E731
            tabV, tabK = one(P // 2 + 1, X), one(P, X // 2 + 1)
            W = torch.ones((P, X), dtype=rt, device="cuda")
            w = torch.ones((1, max(P, X)), dtype=torch.float64, device="cuda")
            obs = torch.empty((2, M), dtype=torch.float64, device="cuda")
            d = _lib.WignerDesc()
            d.W, d.w_bstride, d.step_kind = W.data_ptr(), P * X, _lib.FW_STEP_FUSED
            d.tabV, d.tabK, d.Mx, d.Mp = tabV.data_ptr(), tabK.data_ptr(), 1, 1
            d.wx = d.wp = w.data_ptr()
            d.obs_out, d.dxdp, d.in_scale = obs.data_ptr(), 1.0, 1.0 / (P * X)
            s = torch.cuda.Stream()
            plan = _lib.c_vp()
            _lib.check(lib.fw_wigner_plan_create(P, X, 1, code, ctypes.byref(plan)))
            torch.cuda.synchronize()
            for _ in range(400):
                _lib.check(lib.fw_wigner_propagate(plan, ctypes.byref(d), 2, ctypes.c_void_p(s.cuda_stream)))
            s.synchronize()
            lib.fw_wigner_plan_destroy(plan)
        except Exception as e:
            errors.append(f"P = {P}: {e}")

    threads = [threading.Thread(target=work, args=(P,)) for P in (4096, 128, 4096, 256, 2048, 128)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
