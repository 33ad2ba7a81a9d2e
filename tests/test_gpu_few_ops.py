"""A few ops on a small state: launched one by one, more of them in sweeps.

Below 14 qubits a handful of queued ops costs less as single launches than as
a sweep. Either way the state is the same: bit for bit in exact and f32
arithmetic, within 1e-13 in fast f64 (a dozen double-float steps of 2^-46),
against sweeps whatever the count (the forcing flag).
"""

import numpy as np
import pytest

from helpers import bits_equal, max_delta, rand_matrix, rand_state

pytestmark = pytest.mark.gpu


def unitary(dim, seed):
    return np.ascontiguousarray(np.linalg.qr(rand_matrix(dim, seed))[0])


def apply(be, n, count, seed):
    rng = np.random.default_rng(seed)
    for i in range(count):
        kind = rng.integers(5)
        qs = [int(q) for q in rng.permutation(n)[:2]]
        if kind == 0:
            be.apply_cx(qs[0], qs[1])
        elif kind == 1:
            be.apply_diagonal(sorted(qs), np.exp(1j * rng.uniform(0, 6, 4)))
        elif kind == 2:
            be.apply_unitary(sorted(qs), unitary(4, seed + i))
        else:
            be.apply_unitary(qs[:1], unitary(2, seed + i))


@pytest.mark.parametrize("n", (3, 8, 13))
@pytest.mark.parametrize("prec,flags", ((64, 0), (64, 1), (32, 1), (32, 0)))
def test_same_state_either_way(zc, n, prec, flags):
    for count in (1, 2, 3, 4, 5, 10, 11, 12, 40):
        start = rand_state(n, count, normalize=True)
        got = []
        for extra in (0, zc.FLAG_FORCE_SWEEPS):
            be = zc.CudaBackend(n, prec, flags | extra)
            be.load_state(start)
            apply(be, n, count, 100 * n + count)
            got.append(be.statevector())
            be.close()
        if prec == 64 and flags:
            assert max_delta(*got) < 1e-13, (count, max_delta(*got))
        else:
            assert bits_equal(*got), count


@pytest.mark.parametrize("prec,flags,few", ((64, 0, 1), (64, 1, 10), (32, 1, 3), (32, 0, 3)))
def test_few_ops_are_single_launches(zc, prec, flags, few):
    n = 8
    for count, single in ((1, True), (few, True), (few + 1, False), (few + 40, False)):
        be = zc.CudaBackend(n, prec, flags)
        be.finish()
        before = be.counters()["launches"]
        for i in range(count):
            be.apply_unitary([i % n], unitary(2, i))
        be.finish()
        launches = be.counters()["launches"] - before
        assert launches == count if single else launches < count, (count, launches)
        be.close()
