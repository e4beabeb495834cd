"""fw_wigner_propagate_noalloc and its scratch query on grids of the generic passes:
either length, or both, no power of two (the query once divided by zero there)."""
import ctypes

import pytest

from fastwigner_b200 import _lib

SIZES = [(128, 96, 3), (96, 128, 3), (98, 202, 1), (6, 4, 2), (100, 250, 40), (512, 24, 5)]


@pytest.mark.parametrize("dtype", [_lib.FW_F32, _lib.FW_F64])
def test_scratch_query_of_every_size(dtype):
    lib = _lib.load()
    for P in list(range(4, 140, 2)) + [256, 998, 4094, 4096]:
        for X in list(range(4, 140, 2)) + [256, 998, 4094, 4096]:
            need = lib.fw_noalloc_scratch_needed(P, X, 1, dtype, None)
            real = 8 if dtype == _lib.FW_F64 else 4
            assert need >= 2 * real * (P + X), (P, X)


@pytest.mark.gpu
@pytest.mark.parametrize("P,X,batch", SIZES)
@pytest.mark.parametrize("observables", [False, True])
@pytest.mark.parametrize("precision,tol", [("float64", 1e-10), ("float32", 1e-5)])
def test_generic_sizes_match_the_plan_entry_point(P, X, batch, observables, precision, tol):
    import torch

    from tests.test_zz_no_alloc import _compare_one_call, _plan, _setup

    lib = _lib.load()
    code = _lib.FW_F64 if precision == "float64" else _lib.FW_F32
    c = _setup(P, X, batch, code)
    W, Wref = c["W"], c["W"].clone()
    plan = _plan(lib, c, code)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    try:
        for _ in range(2):
            _compare_one_call(lib, code, c, plan, W, Wref, observables, tol, stream)
    finally:
        lib.fw_wigner_plan_destroy(plan)
