"""Dense blocks of two to four qubits held in registers, alone and between
sweeps and permutations (which hand the state over as float pairs), over
supports with low, high and middle qubits and states from the block's size.

Exact: the oracle's bits. Fast f64: 1e-12, f32: 1e-5, the bounds of the fast
modes, on unitary blocks.
"""

import numpy as np
import pytest

from helpers import bits_equal, rand_matrix, rand_state

pytestmark = pytest.mark.gpu


def unitary(dim, seed):
    return np.linalg.qr(rand_matrix(dim, seed))[0]


@pytest.mark.parametrize("prec,fast", ((64, 0), (64, 1), (32, 0), (32, 1)))
@pytest.mark.parametrize("k", (2, 3, 4))
@pytest.mark.parametrize("extra", (0, 1, 5, 11))
def test_blocks_between_sweeps(zc, oracle, extra, k, prec, fast):
    n = k + extra
    supports = [list(range(k)), list(range(n - k, n)), sorted({0, n - 1, *range(n // 2, n // 2 + k)})[:k]]
    rng = np.random.default_rng(100 * extra + k)
    supports += [sorted(int(x) for x in rng.choice(n, k, replace=False)) for _ in range(3)]
    supports = [s for s in supports if len(s) == k and s[-1] < n]
    amps = rand_state(n, n, normalize=True)
    g, o = zc.CudaBackend(n, prec, zc.FLAG_FAST if fast else zc.FLAG_EXACT), oracle.State(n, prec)
    g.load_state(amps)
    o.load(amps)
    for i, qs in enumerate(supports):
        m = unitary(1 << k, 31 * n + i)
        g.apply_unitary(qs, m)
        o.apply_unitary(qs, m)
        if i % 3 == 0:  # gates on both sides: a sweep
            for q in (0, n - 1):
                h = unitary(2, i + q)
                g.apply_unitary([q], h)
                o.apply_unitary([q], h)
        elif i % 3 == 1:  # a permutation alone
            g.apply_cx(0, n - 1)
            o.apply_cx(0, n - 1)
    a, b = g.statevector(), o.statevector()
    if fast:
        assert np.abs(a - b).max() <= (1e-12 if prec == 64 else 1e-5)
    else:
        assert bits_equal(a, b)
    g.close()
