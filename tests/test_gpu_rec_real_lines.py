"""Even lines of real values through the reconstruction's transforms: the mean and the
middle mode are real, and come out with an imaginary part of exactly 0, so that the
phase which the reconstruction takes of them is 0 or pi and never minus pi by the sign
of a rounding error."""
import numpy as np
import pytest

import mat3d_b200 as m3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", [18, 20, 30, 36, 50, 54, 60, 90, 126, 150, 162, 198, 234, 342])
def test_real_modes(n, axis):
    x = np.random.default_rng(n).standard_normal(n)
    shape = [1, 1, 1]
    shape[axis] = n
    X = m3d.fft3(x, shape)
    assert X[0].imag == 0 and X[n // 2].imag == 0
    assert np.allclose(X, np.fft.fft(x), rtol=0, atol=1e-12 * np.abs(x).sum())
