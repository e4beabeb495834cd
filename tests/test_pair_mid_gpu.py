"""The paired spectral mid-point (pair_mid) at every register-resident length,
in either axis and precision, one instance (small launch shapes) and several,
a single step (two half-steps of their own) and fused ones: states and every
observable sum against the FP64 oracle at the tolerances of the other
propagator tests (1e-10 FP64, 1e-5 FP32)."""
import numpy as np
import pytest

from oracle.wigner_oracle import WignerOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,X", [(128, 4096), (256, 2048), (512, 128), (1024, 256), (2048, 512), (4096, 1024)])
@pytest.mark.parametrize("precision,tol", [("float64", 1e-10), ("float32", 1e-5)])
@pytest.mark.parametrize("batch,steps", [(1, 1), (4, 3)])
def test_states_and_sums(P, X, precision, tol, batch, steps):
    from fastwigner_b200.batch import WignerMoyalBatch

    V = lambda x: 0.05 * x ** 4 - x ** 2  # noqa: E731
    K = lambda p: 0.5 * p ** 2  # noqa: E731
    dV, dK = lambda x: 0.2 * x ** 3 - 2 * x, lambda p: p  # noqa: E731
    kw = dict(X_gridDIM=X, X_amplitude=6.0, P_gridDIM=P, P_amplitude=6.0, dt=0.01)
    b = WignerMoyalBatch(batch=batch, V=V, K=K, diff_V=dV, diff_K=dK, precision=precision, **kw)
    rng = np.random.default_rng(P + X)
    W0 = np.stack([np.exp(-(b.X - rng.uniform(-2, 2)) ** 2 - (b.P - rng.uniform(-1, 1)) ** 2) for _ in range(batch)])
    b.set_wignerfunctions(W0)
    obs = b.propagate(steps).cpu().numpy()
    W = b.W.double().cpu().numpy()
    i = batch - 1
    o = WignerOracle(t=0.0, V=V, K=K, diff_V=dV, diff_K=dK, **kw)
    o.set_wignerfunction(W0[i])
    o.propagate(steps)
    assert np.linalg.norm(W[i] - o.W) / np.linalg.norm(o.W) < tol
    S = obs[:, i, 0]
    for q, ref, sgn in ((2, "X_average", 1), (3, "P_average_RHS", -1), (5, "P_average", 1), (6, "X_average_RHS", 1)):
        np.testing.assert_allclose(sgn * obs[:, i, q] / S, getattr(o, ref), rtol=100 * tol, atol=100 * tol)
    np.testing.assert_allclose((obs[:, i, 4] + obs[:, i, 7]) / S, o.hamiltonian_average, rtol=100 * tol, atol=100 * tol)
    np.testing.assert_allclose(obs[-1, i, 1] / S[-1] ** 2, (o.W ** 2).sum() / o.W.sum() ** 2, rtol=100 * tol)
