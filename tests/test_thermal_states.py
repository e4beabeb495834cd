"""Surrogate thermal states against baseline(): the kernel that adds the harmonic
baseline to the network's output, and predict() around it."""
import numpy as np
import pytest
import torch


def _surrogate(grid, x_e=-2.0):
    from fastwigner_b200.fno import BlochSurrogate, FNO2d, MorseBlochSetup

    return BlochSurrogate(MorseBlochSetup(grid=grid, x_e=x_e), net=FNO2d(layers=1, seed=4))


def _want(s, Ds, As, beta, out):
    """predict() from the network's output in FP64 around baseline()."""
    P = np.stack([np.asarray(Ds, dtype=np.float64), np.asarray(As, dtype=np.float64), np.full(len(Ds), beta)], axis=1)
    b = s.baseline(P).double()
    w = b + b.amax(dim=(1, 2), keepdim=True) * out.double()
    S = w.sum(dim=(1, 2), keepdim=True)
    cond = 1 + w.abs().sum(dim=(1, 2), keepdim=True) / S.abs()  # of the normalisation's sum
    return w / (S * s.s.dX * s.s.dP), cond


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [34, 96, 300])
@pytest.mark.parametrize("x_e", [-2.0, 30.0, -150.0])
def test_predict_matches_baseline(grid, x_e):
    """Row counts below 64 and not a multiple of it, columns not a multiple of 256, well
    centres inside the box and far outside it."""
    s = _surrogate(grid, x_e)
    Ds, As, beta = np.array([2.5, 7.0, 9.5]), np.array([0.6, 1.0, 1.4]), 4.0
    got = s.predict(Ds, As, beta, chunk=2)
    from fastwigner_b200.fno import normalise_params

    out = s.net.forward(normalise_params(np.stack([Ds, As, np.full(3, beta)], axis=1)), s.xs, s.ps, cache=False)
    want, cond = _want(s, Ds, As, beta, out)
    assert torch.isfinite(got).all()
    # FP32 baseline, product and sum: a few roundings of the peak
    assert ((got.double() - want).abs() <= 5e-7 * cond * want.abs().amax(dim=(1, 2), keepdim=True)).all()
