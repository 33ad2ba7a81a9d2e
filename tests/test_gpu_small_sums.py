"""Sums and draws of small states, on both sides of the sizes that decide how a
chain is added up (128 elements: of amplitudes, of one qubit's half, of chunk
masses) and how many threads a chunk gets (4096 amplitudes).

Exact mode: norm, P(1) and draws are the oracle's, bit for bit. Fast mode: its
draws are the exact ones (a draw would have to fall within 2^-46 of a boundary
to move).
"""

import numpy as np
import pytest

from helpers import rand_state

pytestmark = pytest.mark.gpu


def amplitudes(n):
    a = rand_state(n, n, normalize=True)
    a[: min(3, len(a) - 1)] = 0.0  # no mass at the front
    return a


@pytest.mark.parametrize("prec", (64, 32))
@pytest.mark.parametrize("n", (1, 2, 4, 5, 6, 7, 8, 9))
def test_short_chains(zc, oracle, n, prec):
    g, o = zc.CudaBackend(n, prec), oracle.State(n, prec)
    g.load_state(amplitudes(n))
    o.load(amplitudes(n))
    assert g.norm_sqr() == o.norm_sqr()
    for q in range(n):
        assert g.prob_one(q) == o.prob_one(q)
    for shots, seed in ((1, 3), (7, 4), (3000, 5)):
        assert np.array_equal(g.sample(shots, seed), o.sample(shots, seed)), (shots, seed)
    g.close()


@pytest.mark.parametrize("n", (22, 23, 24))
def test_chunk_masses(zc, n):
    """2^6 to 2^8 chunk masses, added up one by one."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    g = zc.CudaBackend(n, 64)
    g.load_state(a)
    p = a.real * a.real + a.imag * a.imag
    masses = np.cumsum(p.reshape(-1, 1 << 16), axis=1)[:, -1]  # left to right
    assert g.norm_sqr() == np.cumsum(masses)[-1]
    g.close()


@pytest.mark.parametrize("prec", (64, 32))
@pytest.mark.parametrize("n", (1, 5, 11, 12, 13))
def test_fast_draws(zc, n, prec):
    fast, exact = zc.CudaBackend(n, prec, zc.FLAG_FAST), zc.CudaBackend(n, prec)
    for be in (fast, exact):
        be.load_state(amplitudes(n))
    for shots, seed in ((1, 3), (500, 4)):
        assert np.array_equal(fast.sample(shots, seed), exact.sample(shots, seed)), (shots, seed)
    fast.close()
    exact.close()
