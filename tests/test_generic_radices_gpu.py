"""Every radix of the generic passes (wigner_generic.cu) and the shapes around
them: register radices 2, 3, 4, 5, 7, 8, 11, 13, 16, one and two direct prime
stages in either axis, pair counts that leave the last tile ragged, single
half-steps (one step) and fused ones, against the FP64 oracle at the
tolerances of the other generic-size tests (1e-10 FP64, 1e-5 FP32)."""
import numpy as np
import pytest

from oracle.wigner_oracle import WignerOracle

pytestmark = pytest.mark.gpu

SIZES = [(4, 6), (22, 26), (154, 130), (34, 38), (578, 646), (1154, 98), (4094, 12), (12, 4094), (4096, 36), (36, 16),
         (352, 2048), (810, 1350)]


@pytest.mark.parametrize("P,X", SIZES)
@pytest.mark.parametrize("precision,tol", [("float64", 1e-10), ("float32", 1e-5)])
@pytest.mark.parametrize("batch,steps", [(1, 1), (5, 3)])
def test_batch_matches_oracle(P, X, precision, tol, batch, steps):
    from fastwigner_b200.batch import WignerMoyalBatch

    V = lambda x: 0.05 * x ** 4 - x ** 2  # noqa: E731
    K = lambda p: 0.5 * p ** 2  # noqa: E731
    dV, dK = lambda x: 0.2 * x ** 3 - 2 * x, lambda p: p  # noqa: E731
    kw = dict(X_gridDIM=X, X_amplitude=6.0, P_gridDIM=P, P_amplitude=6.0, dt=0.01)
    b = WignerMoyalBatch(batch=batch, V=V, K=K, diff_V=dV, diff_K=dK, precision=precision, **kw)
    rng = np.random.default_rng(P * 5000 + X)
    W0 = np.stack([np.exp(-(b.X - rng.uniform(-2, 2)) ** 2 - (b.P - rng.uniform(-1, 1)) ** 2) for _ in range(batch)])
    b.set_wignerfunctions(W0)
    obs = b.propagate(steps).cpu().numpy()
    W = b.W.double().cpu().numpy()
    for i in (0, batch - 1):
        o = WignerOracle(t=0.0, V=V, K=K, diff_V=dV, diff_K=dK, **kw)
        o.set_wignerfunction(W0[i])
        o.propagate(steps)
        assert np.linalg.norm(W[i] - o.W) / np.linalg.norm(o.W) < tol
        S = obs[:, i, 0]
        for q, ref, sgn in ((2, "X_average", 1), (3, "P_average_RHS", -1), (5, "P_average", 1),
                            (6, "X_average_RHS", 1)):
            np.testing.assert_allclose(sgn * obs[:, i, q] / S, getattr(o, ref), rtol=100 * tol, atol=100 * tol)
        np.testing.assert_allclose(obs[-1, i, 1] / S[-1] ** 2, (o.W ** 2).sum() / o.W.sum() ** 2, rtol=100 * tol)
