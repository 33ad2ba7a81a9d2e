"""f64 amplitudes enter double-float arithmetic rounded, not truncated.

Diagonals of ones leave a fast f64 state as the conversion to float pairs and
back leaves it (24 bits and 23 more; the way back and the factor are exact):
each component within half a unit of the 47th bit, 2^-47 of it, and no bias -
the mean signed error of 2^15 components is within six of its standard errors,
2^-47 / sqrt(3 * 2^15) each.
"""

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", (0, 4))
def test_round_trip_through_pairs(zc, flags):
    n = 14
    rng = np.random.default_rng(3)
    a = np.exp(rng.uniform(-3, 3, 1 << n)) * rng.choice((-1, 1), 1 << n)
    b = np.exp(rng.uniform(-3, 3, 1 << n)) * rng.choice((-1, 1), 1 << n)
    a[0], b[0] = 1.0 - 2.0**-53, -(2.0 - 2.0**-52)  # round up across a binade
    be = zc.CudaBackend(n, 64, zc.FLAG_FAST | flags)
    be.load_state(a + 1j * b)
    be.apply_diagonal([0], np.ones(2))
    be.apply_diagonal([5], np.ones(2))
    v = be.statevector()
    be.close()
    x, y = np.concatenate([a, b]), np.concatenate([v.real, v.imag])
    e = (y - x) / x
    assert np.abs(e).max() <= 2.0**-47
    away = (np.abs(y) - np.abs(x)) / np.abs(x)  # truncation shrinks every one
    assert abs(away.mean()) <= 6 * 2.0**-47 / math.sqrt(3 * len(x))
    assert v[0].real == 1.0 and v[0].imag == -2.0
