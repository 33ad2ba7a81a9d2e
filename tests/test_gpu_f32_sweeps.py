"""f32 sweeps against one launch per op, bit for bit.

A register pass of an f32 sweep takes a run of gates, diagonals and CX on four
tile bits and rounds each element as the ops one by one do. Bit 0 and the highest tile bit, runs that end early, controls inside and
outside a group and tiles from three qubits to several tiles are in the draw.
The tolerance is none: the bits are the same.
"""

import numpy as np
import pytest

from helpers import bits_equal, rand_matrix, rand_state

pytestmark = pytest.mark.gpu


def draw_ops(kinds, n, count, seed):
    rng = np.random.default_rng(seed)
    ops = []
    for _ in range(count):
        r, s = int(rng.integers(0, 10)), int(rng.integers(1 << 30))
        if "c" in kinds and r < 3:
            ops.append(("cx", [int(x) for x in rng.choice(n, 2, replace=False)], s))
        elif "d" in kinds and r < 5:
            k = int(rng.integers(1, min(n, 5) + 1))
            ops.append(("d", sorted(int(x) for x in rng.choice(n, k, replace=False)), s))
        else:
            ops.append(("u", [int(rng.integers(n))], s))
    return ops


def play(zc, n, ops, flags):
    g = zc.CudaBackend(n, 32, flags)
    g.load_state(rand_state(n, n, normalize=True))
    for kind, qs, s in ops:
        if kind == "cx":
            g.apply_cx(*qs)
        elif kind == "d":
            g.apply_diagonal(qs, rand_state(len(qs), s))
        else:
            g.apply_unitary(qs, rand_matrix(2, s))
    return g.statevector()


# fast states of 14 qubits and more reorder disjoint gates: exact mode there
@pytest.mark.parametrize("n,fast", [(n, f) for n in (3, 4, 5, 9, 12, 13) for f in (0, 1)] + [(14, 0), (16, 0)])
@pytest.mark.parametrize("kinds", ("u", "uc", "ud", "ucd"))
def test_f32_sweep_passes_have_the_bits_of_single_ops(zc, kinds, n, fast):
    mode = zc.FLAG_FAST if fast else zc.FLAG_EXACT
    for seed, count in ((1, 8), (2, 40), (3, 130)):
        ops = draw_ops(kinds, n, count, 100 * n + seed)
        a = play(zc, n, ops, mode | zc.FLAG_FORCE_SWEEPS)
        b = play(zc, n, ops, mode | zc.FLAG_NO_SWEEPS)
        assert bits_equal(a, b), (seed, count)
