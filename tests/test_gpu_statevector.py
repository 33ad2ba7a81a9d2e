"""statevector returns the state bit for bit: below and at one thread's four
amplitudes, and across the staging buffer's edge (2^21 amplitudes)."""

import numpy as np
import pytest

from helpers import as_precision, bits_equal, rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", (64, 32))
@pytest.mark.parametrize("n", (1, 2, 3, 10, 21, 22))
def test_round_trip(zc, prec, n):
    amps = rand_state(n, n)
    amps[0] = -0.0
    amps[-1] = complex(1e-40, -1e30)
    g = zc.CudaBackend(n, prec)
    g.load_state(amps)
    assert bits_equal(g.statevector(), as_precision(amps, prec))
    g.close()
