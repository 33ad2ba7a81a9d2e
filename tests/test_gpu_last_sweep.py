"""A fast f64 sweep that no sweep follows applies its pending diagonals itself.

One-qubit gates are lowered to rotations between diagonals; the diagonals left
at the end go on to the next sweep, where there is one. At the end of the queue
and before a dense block there is none, and they used to take a launch (and
the state's return from float pairs) of their own.
"""

import numpy as np
import pytest

from helpers import max_delta, rand_matrix, rand_state

pytestmark = pytest.mark.gpu


def unitary(dim, seed):
    return np.ascontiguousarray(np.linalg.qr(rand_matrix(dim, seed))[0])


@pytest.mark.parametrize("n,gates", ((8, 11), (13, 26), (16, 32)))
@pytest.mark.parametrize("dense", (False, True))
def test_one_launch(zc, n, gates, dense):
    states = []
    for flags in (zc.FLAG_FAST, zc.FLAG_EXACT):
        be = zc.CudaBackend(n, 64, flags)
        be.load_state(rand_state(n, n, normalize=True))
        before = be.counters()["launches"]
        for i in range(gates):
            be.apply_unitary([i % min(n, 8)], unitary(2, i))
        if dense:
            be.apply_unitary([0, n - 1], unitary(4, 99))
        be.finish()
        if flags == zc.FLAG_FAST and n <= 8:
            assert be.counters()["launches"] - before == 1 + dense
        states.append(be.statevector())
        be.close()
    # each gate two double-float steps of 2^-46 on each amplitude
    assert max_delta(*states) <= 2 * (gates + 4) * 2.0**-46
