"""statevector writes the caller's array and nothing beside it.

The array's pages are touched before the device writes them: at any offset
within a page, below and across the staging buffer's edge (2^21 amplitudes),
the result is the state bit for bit and the words around the array stay.
"""

import ctypes

import numpy as np
import pytest

from helpers import as_precision, bits_equal, rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", (64, 32))
@pytest.mark.parametrize("n,offset", ((1, 0), (3, 16), (12, 4080), (13, 65536 - 16), (21, 32), (22, 16)))
def test_only_the_array(zc, n, prec, offset):
    amps = rand_state(n, n)
    g = zc.CudaBackend(n, prec)
    g.load_state(amps)
    guard = 8
    raw = np.full((2 << n) + 2 * guard + (1 << 14), 7.25)
    start = (65536 - raw.ctypes.data % 65536) % 65536 // 8 + offset // 8 % (1 << 13)
    lo = start if start >= guard else guard
    out = raw[lo : lo + (2 << n)]
    assert zc.load().zc_statevector(g._h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    assert bits_equal(out.view(np.complex128), as_precision(amps, prec))
    assert (raw[:lo] == 7.25).all() and (raw[lo + (2 << n) :] == 7.25).all()
    g.close()
