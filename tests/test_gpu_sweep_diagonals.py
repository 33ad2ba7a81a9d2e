"""Table diagonals of a sweep, in register passes (up to eight qubits) and on
their own: one to twelve qubits, supports inside a tile, outside it and across,
states from under one warp's elements to many tiles. Exact: the oracle's bits.
Fast: 1e-12 (f64) and 1e-5 (f32) on unit-modulus tables.
"""

import numpy as np
import pytest

from helpers import bits_equal, rand_matrix, rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,fast", ((64, 0), (64, 1), (32, 0), (32, 1)))
@pytest.mark.parametrize("n", (3, 4, 8, 10, 12, 13, 16))
def test_diagonals_in_sweeps(zc, oracle, n, prec, fast):
    rng = np.random.default_rng(n)
    amps = rand_state(n, n, normalize=True)
    g, o = zc.CudaBackend(n, prec, zc.FLAG_FAST if fast else zc.FLAG_EXACT), oracle.State(n, prec)
    g.load_state(amps)
    o.load(amps)
    for k in [k for k in (1, 2, 8, 9, 10, 12) if k <= n] * 2:
        for qs in (sorted(int(x) for x in rng.choice(n, k, replace=False)), list(range(n - k, n))):
            d = np.exp(2j * np.pi * rng.random(1 << k))
            q, u = int(rng.integers(n)), np.linalg.qr(rand_matrix(2, k + n))[0]
            for s in (g, o):
                s.apply_diagonal(qs, d)
                s.apply_unitary([q], u)
    a, b = g.statevector(), o.statevector()
    if fast:
        assert np.abs(a - b).max() <= (1e-12 if prec == 64 else 1e-5)
    else:
        assert bits_equal(a, b)
    g.close()
