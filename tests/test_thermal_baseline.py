"""predict() uses the object's own baseline(): a subclass or an instance that
replaces it trains and predicts on the same one."""
import types

import numpy as np
import pytest
import torch


def test_rule_of_the_thermal_kernel(monkeypatch):
    from fastwigner_b200.fno import BlochSurrogate

    class Sub(BlochSurrogate):
        def baseline(self, P, full=True):
            return None

    def make(cls, G):
        s = cls.__new__(cls)
        s.s = types.SimpleNamespace(G=G)
        return s

    assert make(BlochSurrogate, 16384)._thermal_kernel()
    assert not make(BlochSurrogate, 16386)._thermal_kernel()  # rows past the kernel's
    assert not make(Sub, 512)._thermal_kernel()
    s = make(BlochSurrogate, 512)
    s.baseline = lambda P, full=True: None
    assert not s._thermal_kernel()
    monkeypatch.setattr(BlochSurrogate, "baseline", lambda self, P, full=True: None)
    assert not make(BlochSurrogate, 512)._thermal_kernel()


@pytest.mark.gpu
def test_predict_follows_an_overridden_baseline():
    from fastwigner_b200.fno import BlochSurrogate, FNO2d, MorseBlochSetup, normalise_params

    class Flat(BlochSurrogate):
        def baseline(self, P, full=True):
            n, g = len(P), self.s.G if full else self.g
            return torch.full((n, g, g), 1.0 / g ** 2, device="cuda")

    Ds, As, beta = np.array([2.5, 7.0]), np.array([0.6, 1.0]), 4.0
    net = FNO2d(layers=1, seed=4)
    plain = BlochSurrogate(MorseBlochSetup(grid=96), net=net)
    plain.baseline = lambda P, full=True: torch.full((len(P), 96, 96), 1.0 / 96 ** 2, device="cuda")
    for s in (Flat(MorseBlochSetup(grid=96), net=net), plain):
        out = net.forward(normalise_params(np.stack([Ds, As, np.full(2, beta)], axis=1)), s.xs, s.ps, cache=False)
        w = 1.0 / 96 ** 2 * (1 + out.double())
        S = w.sum(dim=(1, 2), keepdim=True)
        want = w / (S * s.s.dX * s.s.dP)
        cond = 1 + w.abs().sum(dim=(1, 2), keepdim=True) / S.abs()
        assert ((s.predict(Ds, As, beta).double() - want).abs() <= 5e-7 * cond * want.abs().amax(dim=(1, 2), keepdim=True)).all()
