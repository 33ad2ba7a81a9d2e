"""Exact-mode sums where their parallel evaluation can go wrong.

norm_sqr, prob_one and sampled indices must equal the oracle's serial f64
sums bit for bit: tile and row edges (a tile is 2048 elements, a row 32),
masses full of ties (equal amplitudes, powers of two), zeros between
masses, subnormal masses, and infinite or NaN amplitudes.
"""

import numpy as np
import pytest

from helpers import rand_state

pytestmark = pytest.mark.gpu


def states(n, seed):
    rng = np.random.default_rng(seed)
    N = 1 << n
    yield "random", rand_state(n, seed, normalize=True)
    yield "uniform", np.full(N, 2.0 ** (-n / 2.0), complex)
    yield "powers", np.ldexp(1.0, -rng.integers(0, 30, N)) * (1 + 0j)
    yield "sparse", rand_state(n, seed) * (rng.integers(0, 9, N) == 0)
    late = np.zeros(N, complex)
    late[-1] = 0.5 + 0.25j
    yield "last", late


def same(a, b):
    return np.float64(a).tobytes() == np.float64(b).tobytes() or (np.isnan(a) and np.isnan(b))


@pytest.mark.parametrize("prec", (64, 32))
@pytest.mark.parametrize("n", (1, 4, 5, 6, 10, 11, 12, 13, 16, 17, 18))
def test_sums_and_samples(zc, oracle, prec, n):
    g, o = zc.CudaBackend(n, prec), oracle.State(n, prec)
    for what, amps in states(n, 40 + n):
        g.load_state(amps)
        o.load(amps)
        assert same(g.norm_sqr(), o.norm_sqr()), what
        for q in {0, n // 2, n - 1}:
            assert same(g.prob_one(q), o.prob_one(q)), (what, q)
        for shots in (1, 700):
            assert np.array_equal(g.sample(shots, 3), o.sample(shots, 3)), (what, shots)
    g.close()


def test_odd_values(zc, oracle):
    n = 13
    for what, at in (("subnormal", 1e-160), ("huge", 1e200), ("inf", np.inf), ("nan", np.nan)):
        amps = rand_state(n, 5) * (1e-158 if what == "subnormal" else 1.0)
        amps[3000] = at
        g, o = zc.CudaBackend(n, 64), oracle.State(n, 64)
        g.load_state(amps)
        o.load(amps)
        assert same(g.norm_sqr(), o.norm_sqr()), what
        assert same(g.prob_one(12), o.prob_one(12)), what
        g.close()
