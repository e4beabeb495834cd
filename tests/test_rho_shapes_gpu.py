"""Density-matrix steps at every transform length and precision, with static
observables (their kernels in the state precision) and time-dependent ones,
against plain FP64 torch: states at 1e-10 / 1e-5 relative, Ehrenfest lists at
100 times that of the largest value (their sums run over N^2 rounded elements;
the energy, whose kinetic weights reach 1e5, is left to the FP64 fixtures)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("precision,tol", [("float64", 1e-10), ("float32", 1e-5)])
@pytest.mark.parametrize("driven", [False, True])
def test_steps_match_torch(N, precision, tol, driven):
    from fastwigner_b200 import RhoVNeumannCUDA1D

    if driven and N > 1024:
        pytest.skip("the driven case differs only in where the observable kernels come from")
    dt, A, steps = 0.01, 8.0, 3
    V = "0.05 * X * X * X * X - X * X" + (" + 0.3 * X * sin(t)" if driven else "")
    q = RhoVNeumannCUDA1D(X_gridDIM=N, X_amplitude=A, dt=dt, t=0.0, K="0.5 * P * P", V=V, diff_K="P",
                          diff_V="0.2 * X * X * X - 2.0 * X" + (" + 0.3 * sin(t)" if driven else ""),
                          precision=precision)
    dX = 2 * A / N
    x = torch.arange(N, device="cuda", dtype=torch.float64).sub(N / 2).mul(dX)
    p = torch.fft.fftfreq(N, dX / (2 * np.pi), device="cuda", dtype=torch.float64)
    psi = torch.exp(-2 * (x - 0.7) ** 2 + 0.4j * x)
    rho = psi[:, None] * psi.conj()[None, :]
    q.set_rho(rho)
    got = q.propagate(steps).tensor.to(torch.complex128)
    rho = rho / (rho.diagonal().sum() * dX)
    lists = {k: [] for k in ("X_average", "P_average", "P_average_RHS")}
    uK = torch.exp(-0.5j * dt * p * p)
    for k in range(steps):
        t = (k + 1) * dt
        v = 0.05 * x ** 4 - x ** 2 + (0.3 * x * np.sin(t) if driven else 0.0)
        dv = 0.2 * x ** 3 - 2 * x + (0.3 * np.sin(t) if driven else 0.0)
        u = torch.exp(-0.5j * dt * v)
        eV = u[None, :] * u.conj()[:, None]
        rho = eV * torch.fft.ifft2(torch.fft.fft2(rho * eV) * (uK[None, :] * uK.conj()[:, None]))
        tr = rho.diagonal().sum()
        d = rho.diagonal() / tr
        mom = torch.fft.ifft(torch.fft.fft(rho, dim=1) * p, dim=1).diagonal().sum() / tr
        lists["X_average"].append((d * x).sum().real)
        lists["P_average"].append(mom.real)
        lists["P_average_RHS"].append(-(d * dv).sum().real)
        rho = rho / (tr * dX)
    assert (got - rho).norm() / rho.norm() < tol
    for name, ref in lists.items():
        r = torch.stack(ref).cpu().numpy()
        np.testing.assert_allclose(getattr(q, name), r, rtol=0, atol=100 * tol * max(1.0, np.abs(r).max()))
