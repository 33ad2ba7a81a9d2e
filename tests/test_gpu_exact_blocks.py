"""Exact f64 blocks of four qubits on both sides of the size that decides their
kernel, and larger ones: the oracle's bits."""

import numpy as np
import pytest

from helpers import bits_equal, rand_matrix, rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", ((4, 4), (5, 4), (12, 4), (21, 4), (22, 4), (5, 5), (9, 6), (13, 7)))
def test_exact_blocks(zc, oracle, n, k):
    rng = np.random.default_rng(n + k)
    amps = rand_state(n, n, normalize=True)
    amps[0] = 0.0
    g, o = zc.CudaBackend(n, 64), oracle.State(n, 64)
    g.load_state(amps)
    o.load(amps)
    for qs in (list(range(k)), list(range(n - k, n)), sorted(int(x) for x in rng.choice(n, k, replace=False))):
        m = np.linalg.qr(rand_matrix(1 << k, int(rng.integers(1000))))[0]
        m[0, 0] = 0.0
        g.apply_unitary(qs, m)
        o.apply_unitary(qs, m)
    assert bits_equal(g.statevector(), o.statevector())
    g.close()
