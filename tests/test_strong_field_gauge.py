"""A StrongFieldWigner whose gauge changes between calls: every chunk's field
factors are taken over the axis of the gauge it runs in."""
import types

import numpy as np
import pytest
import torch

from fastwigner_b200.strong_field import StrongFieldWigner


def test_factors_follow_the_axis_they_are_asked_for():
    ns = types.SimpleNamespace(device=torch.device("cpu"), _rt=torch.float64)
    f = np.array([0.3, -1.7, 2.5])
    for axis, c in ((np.linspace(-4, 4, 9), -0.01), (np.linspace(-3, 3, 17), 0.005), (np.linspace(-1, 1, 9), 0.02)):
        for a in (axis, 2 * axis):
            got = torch.view_as_complex(StrongFieldWigner._field_factors(ns, f, a[np.newaxis, :], c)).numpy()
            # FP64 rounding of the phase, its sine and cosine
            np.testing.assert_allclose(got, np.exp(1j * c * np.outer(f, a)), rtol=0, atol=1e-15)


@pytest.mark.gpu
@pytest.mark.parametrize("P,X", [(128, 256), (256, 128), (96, 130)])
@pytest.mark.parametrize("first", ["velocity", "length"])
def test_gauge_switched_between_calls(P, X, first):
    kw = dict(X_gridDIM=X, X_amplitude=8.0, P_gridDIM=P, P_amplitude=4.0, dt=0.01, t=0.0, precision="float64",
              V=lambda self, x: -1.0 / np.sqrt(x ** 2 + 1.5), diff_V=lambda self, x: x / (x ** 2 + 1.5) ** 1.5,
              A=lambda self, t: 0.2 * np.sin(0.7 * t), E=lambda self, t: -0.14 * np.cos(0.7 * t))
    second = "length" if first == "velocity" else "velocity"
    a = StrongFieldWigner(gauge=first, **kw)
    W0 = np.exp(-(a.X - 0.5) ** 2 - (a.P + 0.2) ** 2)
    a.set_wignerfunction(W0)
    a.propagate(3)
    mid = np.array(a.propagate(2))
    a.gauge = second
    got = np.array(a.propagate(4))
    b = StrongFieldWigner(gauge=second, **{**kw, "t": a.t - 4 * a.dt})
    b.set_wignerfunction(mid)
    want = np.array(b.propagate(4))
    # the same kernels on the same factors, up to the rounding of t
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 1e-12
