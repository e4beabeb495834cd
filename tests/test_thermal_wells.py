"""Well parameters of the surrogate's thermal states: FP64 whatever the caller's type, as
in baseline()."""
import numpy as np
import pytest
import torch


def test_well_exponents_in_fp64_whatever_the_input():
    from fastwigner_b200.fno import BlochSurrogate

    Ds, As, beta = [2.7, 9.1], [0.55, 1.4], 3.0
    want = BlochSurrogate._wells(np.array(Ds, dtype=np.float32).astype(np.float64),
                                 np.array(As, dtype=np.float32).astype(np.float64), beta)
    got = BlochSurrogate._wells(np.array(Ds, dtype=np.float32), np.array(As, dtype=np.float32), beta)
    assert got.dtype == np.float64
    np.testing.assert_array_equal(got, want)
    w = np.float64(np.float32(As[0])) * np.sqrt(2 * np.float64(np.float32(Ds[0])))
    np.testing.assert_allclose(want[0], [w, 2 / w * np.tanh(0.5 * beta * w)], rtol=1e-15)
    np.testing.assert_array_equal(BlochSurrogate._wells(np.array([2, 9]), np.array([1, 2]), 3),
                                  BlochSurrogate._wells(np.array([2.0, 9.0]), np.array([1.0, 2.0]), 3.0))
    np.testing.assert_array_equal(BlochSurrogate._wells(Ds, As, [beta, beta]), BlochSurrogate._wells(Ds, As, beta))


@pytest.mark.gpu
def test_predict_takes_fp32_parameters_as_fp64():
    from fastwigner_b200.fno import BlochSurrogate, FNO2d, MorseBlochSetup

    s = BlochSurrogate(MorseBlochSetup(grid=96), net=FNO2d(layers=1, seed=4))
    Ds, As = np.array([2.7, 9.1], dtype=np.float32), np.array([0.55, 1.4], dtype=np.float32)
    assert torch.equal(s.predict(Ds, As, 3.0), s.predict(Ds.astype(np.float64), As.astype(np.float64), 3.0))
