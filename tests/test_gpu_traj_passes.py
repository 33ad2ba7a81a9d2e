"""Trajectory passes over every operand position and state size.

A random circuit followed by its inverse ends in |0...0>, so every shot must
read zero in every qubit. The noise model (readout flips 1 -> 0 only, which
act on no zero) sends the run to the batched engine without changing the
state. Sizes cover each launch shape and its edges (states below five
qubits, shared-memory states, states split with global memory); operands
cover qubits 0 and 1 (lanes of a vector) alone and together, the highest
qubits, one- and two-qubit gates with one entry per row and dense, and
three-qubit gates. A measured and reset qubit in between checks the outcome
and collapse passes.
"""

import numpy as np
import pytest

from zeno_gb300 import circuit as C

pytestmark = pytest.mark.gpu

INVERSE = {"h": "h", "x": "x", "z": "z", "s": "sdg", "t": "tdg", "cx": "cx", "cz": "cz", "swap": "swap", "ccx": "ccx",
           "rx": "rx", "ry": "ry", "rz": "rz", "cp": "cp", "crx": "crx", "rxx": "rxx", "u3": "u3"}


def inverse(name, ps):
    if name == "u3":
        return name, (-ps[0], -ps[2], -ps[1])
    return INVERSE[name], tuple(-p for p in ps)


def circuit(n, seed):
    rng = np.random.default_rng(seed)
    ang = lambda k: tuple(float(x) for x in rng.uniform(0, 6.28, k))  # noqa: E731
    out = [("u3", (q,), ang(3)) for q in range(n)]
    pairs = [(a, b) for a in {0, 1, min(2, n - 1), n - 1} for b in {0, 1, n - 2, n - 1} if a != b]
    for a, b in pairs:
        out += [("cx", (a, b), ()), ("swap", (a, b), ()), ("cp", (a, b), ang(1)), ("crx", (a, b), ang(1)),
                ("rxx", (b, a), ang(1))]
    for q in {0, 1, min(2, n - 1), n - 1}:
        out += [("h", (q,), ()), ("t", (q,), ()), ("x", (q,), ()), ("rx", (q,), ang(1))]
    if n >= 3:
        out += [("ccx", (0, n - 1, 1), ()), ("ccx", (n - 1, n - 2, 0), ())]
    return out


def key_zero(r):
    return all(set(k) <= {"0", " "} for k in r.counts)


@pytest.mark.parametrize("n", (1, 2, 3, 4, 5, 6, 10, 11, 13, 14, 15, 16))
def test_circuit_and_inverse(zc, n):
    gates = circuit(n, n) if n > 1 else [("u3", (0,), (0.3, 1.0, 2.0)), ("h", (0,), ()), ("t", (0,), ())]
    p = C.Program(n, [("c", n)], [])
    for name, qs, ps in gates:
        p.instrs.append(C.Instr(C.I_GATE, name, qs, ps))
    for name, qs, ps in reversed(gates):
        name, ps = inverse(name, ps)
        p.instrs.append(C.Instr(C.I_GATE, name, qs, ps))
    p.instrs += [C.Instr(C.I_MEASURE, qubits=(q,), clbit=q) for q in range(n)]
    r = zc.run(p, shots=40, seed=3, precision=32, noise=zc.NoiseModel(readout_flip_1to0=0.5))
    assert r.batched and sum(r.counts.values()) == 40
    assert key_zero(r), r.counts


@pytest.mark.parametrize("n", (2, 5, 12, 15))
def test_measure_and_reset_between(zc, n):
    """Qubit q is put into |1> and measured (always 1), a condition on that
    bit undoes another qubit's X, q is reset; everything ends in |0>."""
    p = C.Program(n, [("m", 1), ("c", n)], [])
    for q in range(n):
        o = (q + 1) % n
        p.instrs += [C.Instr(C.I_GATE, "x", (q,)), C.Instr(C.I_GATE, "x", (o,)),
                     C.Instr(C.I_MEASURE, qubits=(q,), clbit=0),
                     C.Instr(C.I_GATE, "x", (o,), (), 0, 0, 1),   # runs: the bit is 1
                     C.Instr(C.I_GATE, "h", (o,), (), 0, 0, 0),   # does not
                     C.Instr(C.I_RESET, qubits=(q,))]
    p.instrs += [C.Instr(C.I_MEASURE, qubits=(q,), clbit=1 + q) for q in range(n)]
    r = zc.run(p, shots=300, seed=5, precision=32)
    assert r.batched
    assert set(r.counts) == {"0" * n + " 1"}, r.counts
