"""norm_sqr and prob_one of fast states: below one vector, one CTA, a partly
filled last CTA and several CTAs, qubits inside a vector and above it, twice in
a row (the launch's ticket starts over). Double-float sums: 1e-12 relative.

And the sampling entry point that allocates nothing, on a small state whose
gates are still queued: it draws what the flushed state draws.
"""

import math

import numpy as np
import pytest

from helpers import as_precision, rand_matrix, rand_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", (64, 32))
@pytest.mark.parametrize("n", (1, 2, 3, 4, 9, 10, 11, 13, 20))
def test_fast_totals(zc, prec, n):
    amps = as_precision(rand_state(n, 40 + n), prec)
    p = np.abs(amps.astype(np.complex128).real) ** 2 + np.abs(amps.astype(np.complex128).imag) ** 2
    g = zc.CudaBackend(n, prec, zc.FLAG_FAST)
    g.load_state(amps)
    whole = math.fsum(p)
    for _ in range(2):
        assert abs(g.norm_sqr() - whole) <= 1e-12 * whole
        for q in sorted({0, 1 % n, 2 % n, n // 2, n - 1}):
            ones = math.fsum(p.reshape(-1, 2, 1 << q)[:, 1].ravel())
            assert abs(g.prob_one(q) - ones) <= 1e-12 * whole, q
    g.close()


@pytest.mark.parametrize("prec,n", [(p, n) for p in (64, 32) for n in (1, 11, 12, 13, 16, 18)] + [(32, 25)])
def test_fast_sampler_tiles(zc, prec, n):
    """Chunks below, at and above one tile of the rescan, few chunks (wide CTAs)
    and many: at least 99.9% of 4096 draws are exact mode's."""
    amps = rand_state(n, 70 + n, normalize=True)
    draws = []
    for flags in (zc.FLAG_FAST, zc.FLAG_EXACT):
        g = zc.CudaBackend(n, prec, flags)
        g.load_state(amps)
        draws.append(g.sample(4096, 5))
        g.close()
    assert np.mean(draws[0] == draws[1]) >= 0.999


@pytest.mark.parametrize("prec", (64, 32))
@pytest.mark.parametrize("n", (3, 9, 13))
def test_noalloc_sampler_sees_queued_gates(zc, prec, n):
    a, b = (zc.CudaBackend(n, prec) for _ in range(2))
    for s in (a, b):
        s.load_state(rand_state(n, n, normalize=True))
        for q in range(n):
            s.apply_unitary([q], np.linalg.qr(rand_matrix(2, q))[0])
        s.apply_cx(0, n - 1)
    b.finish()
    assert np.array_equal(a.sample_noalloc(500, 3), b.sample(500, 3))
