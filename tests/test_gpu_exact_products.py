"""Exact f64 gates keep the reference's bits where products leave the common
range: zeros of either sign, subnormals, results that underflow or overflow,
infinities and NaN (a NaN has to be one on both sides; its payload is not
compared), under matrices with zero entries (u3, H, RX, X, a row of zeros) and
diagonals, one launch per op and in sweeps.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = np.array([0.0, -0.0, 5e-324, -2.3e-308, 1e-200, -1e-160, 1.0, -1.5, 3e150, -1e300, np.inf, -np.inf, np.nan,
                  1 + 2.0**-52, 2.0**-537, 2.0**-511])

MATS = {
    "u3": [[0.8, -0.6 + 0.1j], [0.3j, 0.5 - 0.2j]],
    "h": [[2**-0.5, 2**-0.5], [2**-0.5, -(2**-0.5)]],
    "rx": [[0.6, -0.8j], [-0.8j, 0.6]],
    "x": [[0, 1], [1, 0]],
    "row": [[0, 0], [1e-170, 1e200j]],
    "small": [[1e-300, 1e-320], [5e-324j, 1]],
    "inf": [[np.inf, 1], [1, 0.5]],
}


def same(a, b):
    x, y = a.view(np.float64), b.view(np.float64)
    nan = np.isnan(x)
    return np.array_equal(nan, np.isnan(y)) and np.array_equal(x.view(np.uint64)[~nan], y.view(np.uint64)[~nan])


def amplitudes(n, finite):
    rng = np.random.default_rng(n)
    pool = EDGES[np.isfinite(EDGES)] if finite else EDGES
    v = np.empty(2 << n)
    v[:] = rng.choice(pool, 2 << n)
    half = rng.random(2 << n) < 0.5  # ordinary neighbours beside the edges
    v[half] = rng.uniform(-1, 1, int(half.sum()))
    return v.view(np.complex128)


@pytest.mark.parametrize("finite", (True, False))
@pytest.mark.parametrize("n", (2, 5, 9))
@pytest.mark.parametrize("name", sorted(MATS))
def test_edge_values(zc, oracle, name, n, finite):
    m = np.array(MATS[name], complex)
    amps = amplitudes(n, finite)
    with np.errstate(all="ignore"):
        for flags in (zc.FLAG_NO_SWEEPS, zc.FLAG_FORCE_SWEEPS):
            for q in (0, n - 1):
                g, o = zc.CudaBackend(n, 64, flags), oracle.State(n, 64)
                g.load_state(amps)
                o.load(amps)
                for _ in range(2):
                    g.apply_unitary([q], m)
                    o.apply_unitary([q], m)
                    g.apply_diagonal([n - 1 - q], np.diag(m).copy())
                    o.apply_diagonal([n - 1 - q], np.diag(m).copy())
                assert same(g.statevector(), o.statevector()), (flags, q)
                g.close()
