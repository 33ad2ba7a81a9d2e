"""A few ops on a small state.

Below 14 qubits fewer than four queued ops of an f32 state are launched one by
one, and two to seven of a fast f64 state (dense blocks apart) run in exact
arithmetic, where that is faster than a sweep. Bit for bit: f32 states are
those of sweeps whatever the count (the forcing flag), fast f64 states are
exact-mode ones between the two counts and those of sweeps outside them.
"""

import numpy as np
import pytest

from helpers import bits_equal, rand_matrix, rand_state

pytestmark = pytest.mark.gpu


def unitary(dim, seed):
    return np.ascontiguousarray(np.linalg.qr(rand_matrix(dim, seed))[0])


def apply(be, n, count, seed, dense):
    rng = np.random.default_rng(seed)
    for i in range(count):
        kind = rng.integers(5)
        qs = [int(q) for q in rng.permutation(n)[:2]]
        if kind == 0:
            be.apply_cx(qs[0], qs[1])
        elif kind == 1:
            be.apply_diagonal(sorted(qs), np.exp(1j * rng.uniform(0, 6, 4)))
        elif kind == 2 and dense:
            be.apply_unitary(sorted(qs), unitary(4, seed + i))
        else:
            be.apply_unitary(qs[:1], unitary(2, seed + i))


def state(zc, n, prec, flags, count, dense):
    be = zc.CudaBackend(n, prec, flags)
    be.load_state(rand_state(n, count, normalize=True))
    before = be.counters()["launches"]
    apply(be, n, count, 100 * n + count, dense)
    be.finish()
    launches = be.counters()["launches"] - before
    v = be.statevector()
    be.close()
    return v, launches


@pytest.mark.parametrize("n", (1, 2, 3, 8, 13, 14))
@pytest.mark.parametrize("flags", (0, 1))
def test_f32(zc, n, flags):
    for count in (1, 2, 3, 4, 5, 40) if n > 1 else (0,):
        a, launches = state(zc, n, 32, flags, count, True)
        b, _ = state(zc, n, 32, flags | zc.FLAG_FORCE_SWEEPS, count, True)
        assert n == 14 or bits_equal(a, b), count
        assert launches == count if count < 4 and n < 14 else launches <= count


@pytest.mark.parametrize("n", (3, 8, 13, 14))
@pytest.mark.parametrize("dense", (False, True))
def test_fast_f64(zc, n, dense):
    for count in (1, 2, 3, 7, 8, 9, 40):
        few = 2 <= count < 8 and n < 14 and not dense
        fast, _ = state(zc, n, 64, zc.FLAG_FAST, count, dense)
        same, _ = state(zc, n, 64, zc.FLAG_EXACT if few else zc.FLAG_FAST | zc.FLAG_FORCE_SWEEPS, count, dense)
        # (a draw of the dense kind may hold no dense block)
        assert bits_equal(fast, same) or (dense and count < 8), count
