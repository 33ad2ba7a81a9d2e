"""The work that users of the backend have it do, as cases that can be timed.

Four ways of use, each through the package's public entry points:

  run      `backend.run` on a compiled program: one whole call with its counts
           and final state vector (`zeno run --backend cuda`)
  circuit  a `CudaBackend` that a program keeps: reset, apply a compiled
           circuit op by op, read every qubit's P(1), sample; the state,
           gigabytes at the larger sizes, stays on the device as in real use
  noisy    `backend.run` with a noise model or a dynamic circuit: batched
           f32 trajectories, one shot each
  serve    a `Server` that works off a batch of mixed requests

Circuits are the workloads this repository is benchmarked on: u3 layers with
CX on a random matching, the QFT with its SWAP network, and the random gate
mix. `exact` simulates the same gates with plain torch in 64 bits.

Values read from an f32 state (its amplitudes and probabilities) are returned
as f32 numbers, the type they are held in on the device.
"""

import math
import random

import numpy as np
import torch

from zeno_gb300 import backend as zb
from zeno_gb300 import circuit as C
from zeno_gb300 import serve as S

TAU = 2.0 * math.pi
NOISE = dict(depolarizing_1q=1e-3, depolarizing_2q=1e-2, amplitude_damping=1e-3, readout_flip_0to1=0.02,
             readout_flip_1to0=0.02)


def listed():
    return [
        # a first circuit, as the README and the tutorial run it: default (exact f64) arithmetic, 1000 shots
        dict(name="run_8q_exact", use="run", circuit="matching", n=8, depth=6, prec=64, fast=False, fusion=1, shots=1000),
        # a small f32 request on its own, below the size at which ops are batched into sweeps
        dict(name="run_13q_f32", use="run", circuit="mix", n=13, depth=30, prec=32, fast=True, fusion=1, shots=500),
        # the 20-qubit benchmark circuit in the default arithmetic
        dict(name="run_20q_exact", use="run", circuit="matching", n=20, depth=12, prec=64, fast=False, fusion=1,
             shots=1024),
        # the same family at an odd width in fast f64 arithmetic
        dict(name="run_19q_fast", use="run", circuit="matching", n=19, depth=12, prec=64, fast=True, fusion=1, shots=1024),
        # the headline circuit (u3 + matching CX, fast f64) on a state far larger than the L2
        dict(name="circuit_27q_fast", use="circuit", circuit="matching", n=27, depth=10, prec=64, fast=True, fusion=1,
             shots=1024),
        # the same in exact arithmetic, with every qubit's probability read in the reference's summation order
        dict(name="circuit_24q_exact", use="circuit", circuit="matching", n=24, depth=4, prec=64, fast=False, fusion=1,
             shots=1024),
        # f32 gate mix, the serving and precision workload, probabilities read (no shots)
        dict(name="circuit_26q_mix_f32", use="circuit", circuit="mix", n=26, depth=30, prec=32, fast=True, fusion=1,
             shots=0),
        # QFT: diagonal ladders and SWAPs, 8192 shots
        dict(name="circuit_25q_qft", use="circuit", circuit="qft", n=25, depth=1, prec=64, fast=True, fusion=1,
             shots=8192),
        # dense fused blocks, as a front end with a wider fusion setting sends them
        dict(name="run_22q_fused3", use="run", circuit="matching", n=22, depth=8, prec=64, fast=True, fusion=3,
             shots=1024),
        # the noise workload: 16 qubits, depth 20, one shot per trajectory
        dict(name="noisy_16q", use="noisy", circuit="matching", n=16, depth=20, dynamic=False, shots=2048),
        # mid-circuit measurement, conditioned gates and resets
        dict(name="dynamic_13q", use="noisy", circuit="dynamic", n=13, depth=6, dynamic=True, shots=1500),
        # a batch of mixed requests, 8 to 22 qubits
        dict(name="serve_24", use="serve", requests=24, n_min=8, n_max=22, stream=0),
    ]


def draw(rng):
    use = rng.choice(("run", "run", "circuit", "circuit", "circuit", "noisy", "serve"))
    if use == "run":
        n = rng.randint(3, 19)
        prec = rng.choice((32, 64))
        kind = rng.choice(("matching", "mix", "qft"))
        return dict(use=use, circuit=kind, n=n, depth=1 if kind == "qft" else rng.randint(2, 12), prec=prec,
                    fast=rng.random() < (0.8 if prec == 32 else 0.5), fusion=rng.choice((1, 1, 2, 3)),
                    shots=int(math.exp(rng.uniform(0.0, math.log(2048)))))
    if use == "circuit":
        n = rng.randint(20, 25)
        prec = rng.choice((32, 64, 64))
        kind = rng.choice(("matching", "mix", "qft"))
        fast = prec == 32 or rng.random() < 0.7
        return dict(use=use, circuit=kind, n=n, depth=1 if kind == "qft" else rng.randint(2, 8 if fast else 3), prec=prec,
                    fast=fast, fusion=rng.choice((1, 1, 1, 2, 4)), shots=0 if prec == 32 else rng.randint(1, 4096))
    if use == "noisy":
        dynamic = rng.random() < 0.3
        n = rng.randint(5, 16)
        return dict(use=use, circuit="dynamic" if dynamic else rng.choice(("matching", "mix")), n=n,
                    depth=rng.randint(2, 6 if dynamic else 12), dynamic=dynamic,
                    shots=int(math.exp(rng.uniform(math.log(64), math.log(2048)))))
    return dict(use=use, requests=rng.randint(4, 24), n_min=8, n_max=rng.randint(12, 21), stream=rng.randint(1, 9999))


# ------------------------------------------------------------------ circuits
#
# A circuit is a list of (name, qubits, parameters); for dynamic circuits
# also ("measure", (q,), (clbit,)), ("reset", (q,), ()) and ("if", (q,),
# (register,)), an X on q where the one-bit register holds 1.


def _mix_layer(r, n, out):
    order = list(range(n))
    r.shuffle(order)
    pos = 0
    while pos < n:
        u, q = r.random(), order[pos]
        pos += 1
        if u < 0.15:
            out.append(("h", (q,), ()))
        elif u < 0.25:
            out.append(("s", (q,), ()))
        elif u < 0.35:
            out.append(("t", (q,), ()))
        elif u < 0.65:
            out.append((r.choice(("rx", "ry", "rz")), (q,), (TAU * r.random(),)))
        elif pos < n:
            out.append(("cx" if u < 0.9 else "cz" if u < 0.95 else "swap", (q, order[pos]), ()))
            pos += 1
        else:
            out.append(("h", (q,), ()))


def _gates(case, seed):
    """The circuit's gates, from the seed alone."""
    r = random.Random(int(seed) * 1000003 + case["n"])
    n, out = case["n"], []
    if case["circuit"] == "qft":
        x = r.getrandbits(n)
        out += [("x", (q,), ()) for q in range(n) if (x >> q) & 1]
        for i in range(n - 1, -1, -1):
            out.append(("h", (i,), ()))
            out += [("cp", (j, i), (math.pi / float(1 << (i - j)),)) for j in range(i - 1, -1, -1)]
        out += [("swap", (k, n - 1 - k), ()) for k in range(n // 2)]
        return out
    for layer in range(case["depth"]):
        if case["circuit"] == "mix":
            _mix_layer(r, n, out)
            continue
        out += [("u3", (q,), (TAU * r.random(), TAU * r.random(), TAU * r.random())) for q in range(n)]
        if case["circuit"] == "dynamic":
            out += [("cx", (q, q + 1), ()) for q in range(layer % 2, n - 1, 2)]
            mq = r.randrange(n)
            out += [("measure", (mq,), (layer,)), ("if", ((mq + 1) % n,), (layer,)), ("reset", (mq,), ())]
            continue
        order = list(range(n))
        r.shuffle(order)
        for k in range(n // 2):
            a, b = order[2 * k], order[2 * k + 1]
            out.append(("cx", (a, b) if r.random() < 0.5 else (b, a), ()))
    return out


def _program(case, seed):
    n = case["n"]
    extra = case["depth"] if case["circuit"] == "dynamic" else 0
    p = C.Program(n, [("m%d" % i, 1) for i in range(extra)] + [("c", n)], [])
    for name, qs, ps in _gates(case, seed):
        if name == "measure":
            p.instrs.append(C.Instr(C.I_MEASURE, qubits=qs, clbit=ps[0]))
        elif name == "reset":
            p.instrs.append(C.Instr(C.I_RESET, qubits=qs))
        elif name == "if":
            p.instrs.append(C.Instr(C.I_GATE, "x", qs, (), 0, ps[0], 1))
        else:
            p.instrs.append(C.Instr(C.I_GATE, name, qs, ps))
    p.instrs += [C.Instr(C.I_MEASURE, qubits=(q,), clbit=extra + q) for q in range(n)]
    return p


def _requests(case):
    """(qubits, depth, shots, precision) of each request: log-uniform widths,
    depths over 4..60, log-uniform shots, one in twenty at f64."""
    out = []
    for i in range(case["requests"]):
        u = (i + 0.5) / case["requests"]
        n = min(case["n_max"], int(case["n_min"] * ((case["n_max"] + 1) / case["n_min"]) ** u))
        j = i + case["stream"]
        out.append((n, 4 + (37 * j) % 57, max(1, int(math.exp(((0.618034 * j) % 1.0) * math.log(8192)))),
                    64 if j % 20 == 7 else 32))
    return out


# ------------------------------------------------------------------ prepare / run


def prepare(case, seed):
    use = case["use"]
    if use == "serve":
        reqs = []
        for i, (n, depth, shots, prec) in enumerate(_requests(case)):
            c = dict(circuit="mix", n=n, depth=depth)
            reqs.append((zb.compile(_program(c, seed * 64 + i), 1), prec, shots, seed * 64 + i))
        return dict(use=use, server=S.Server(pool_bytes=1 << 30), reqs=reqs)
    p = _program(case, seed)
    if use == "noisy":
        noise = None if case["dynamic"] else zb.NoiseModel(**NOISE)
        return dict(use=use, p=p, program=zb.compile(p, 0), noise=noise, shots=case["shots"], seed=seed)
    program = zb.compile(p, case["fusion"])
    st = dict(use=use, p=p, program=program, shots=case["shots"], seed=seed, prec=case["prec"],
              flags=zb.FLAG_FAST if case["fast"] else zb.FLAG_EXACT)
    if use == "circuit":
        st["backend"] = zb.CudaBackend(case["n"], case["prec"], st["flags"])
        st["ops"] = program.ops
    return st


def _shots(raw):
    """The counts as one classical word per shot, ascending."""
    return np.repeat(np.fromiter(raw.keys(), dtype=np.uint64, count=len(raw)),
                     np.fromiter(raw.values(), dtype=np.int64, count=len(raw)))


def run(st):
    use = st["use"]
    if use == "run":
        r = zb.run(st["p"], shots=st["shots"], seed=st["seed"], precision=st["prec"], flags=st["flags"],
                   program=st["program"], statevector=True)
        sv = r.statevector.astype(np.complex64) if st["prec"] == 32 else r.statevector
        return dict(statevector=sv, samples=_shots(r.raw))
    if use == "noisy":
        r = zb.run(st["p"], shots=st["shots"], seed=st["seed"], precision=32, noise=st["noise"], program=st["program"])
        return dict(samples=_shots(r.raw))
    if use == "serve":
        srv = st["server"]
        ids = [(srv.submit(p, prec, shots, seed), shots) for p, prec, shots, seed in st["reqs"]]
        while True:
            status = srv.step()
            if status.active == 0 and status.pending == 0:
                break
        return [srv.take(rid, shots) for rid, shots in ids]
    be = st["backend"]
    be.reset_all()
    for op in st["ops"]:
        if op.kind == zb.OP_UNITARY:
            be.apply_unitary(op.qubits, op.data)
        elif op.kind == zb.OP_DIAG:
            be.apply_diagonal(op.qubits, op.data)
        elif op.kind == zb.OP_CX:
            be.apply_cx(op.a, op.b)
        else:
            be.apply_swap(op.a, op.b)
    out = dict(p1=np.array([be.prob_one(q) for q in range(be.n)], dtype=np.float32 if st["prec"] == 32 else np.float64))
    if st["shots"]:
        out["samples"] = be.sample(st["shots"], st["seed"])
    return out


# ------------------------------------------------------------------ work / exact


def _gate_flops(name):
    """Arithmetic of one gate per amplitude: a general complex 2x2 costs 14,
    a phase 6 (on the amplitudes it touches), a permutation none."""
    if name in ("cx", "swap", "x", "if"):
        return 0.0
    if name in ("s", "t"):
        return 3.0
    if name == "rz":
        return 6.0
    if name in ("cz", "cp"):
        return 1.5
    if name in ("measure", "reset"):
        return 6.0
    if name in ("h", "ry", "rx"):
        return 6.0
    return 14.0


def work(case):
    """The state written once and read once, the results written once, and
    the gates' arithmetic on every amplitude."""
    if case["use"] == "serve":
        b = f = 0.0
        for i, (n, depth, shots, prec) in enumerate(_requests(case)):
            g = _gates(dict(circuit="mix", n=n, depth=depth), i)
            b += 2.0 * 2 ** n * prec / 4 + 8.0 * shots
            f += 2.0 ** n * sum(_gate_flops(x[0]) for x in g)
        return dict(bytes=b, flops=f)
    amps = 2.0 ** case["n"]
    f = amps * sum(_gate_flops(x[0]) for x in _gates(case, 1))
    if case["use"] == "noisy":
        return dict(bytes=case["shots"] * (2.0 * amps * 8 + 8.0), flops=f * case["shots"])
    amp_bytes = case["prec"] / 4
    out = amps * 2 * amp_bytes if case["use"] == "run" else 8.0 * case["n"]
    return dict(bytes=2.0 * amps * amp_bytes + out + 8.0 * case["shots"], flops=f)


def _matrix(name, ps):
    r = 1.0 / math.sqrt(2.0)
    if name == "x":
        return [[0, 1], [1, 0]]
    if name == "h":
        return [[r, r], [r, -r]]
    if name == "s":
        return [[1, 0], [0, 1j]]
    if name == "t":
        return [[1, 0], [0, complex(r, r)]]
    t = ps[0] / 2.0
    if name == "rx":
        return [[math.cos(t), -1j * math.sin(t)], [-1j * math.sin(t), math.cos(t)]]
    if name == "ry":
        return [[math.cos(t), -math.sin(t)], [math.sin(t), math.cos(t)]]
    if name == "rz":
        return [[complex(math.cos(t), -math.sin(t)), 0], [0, complex(math.cos(t), math.sin(t))]]
    phi, lam = ps[1], ps[2]
    e = lambda a: complex(math.cos(a), math.sin(a))  # noqa: E731
    return [[math.cos(t), -e(lam) * math.sin(t)], [e(phi) * math.sin(t), e(phi + lam) * math.cos(t)]]


def _simulate(n, gates):
    """The final state as a complex128 tensor."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = torch.zeros(1 << n, dtype=torch.complex128, device=dev)
    v[0] = 1.0
    for name, qs, ps in gates:
        if len(qs) == 2:
            hi, lo = max(qs), min(qs)
            w = v.view(1 << (n - 1 - hi), 2, 1 << (hi - 1 - lo), 2, 1 << lo)
            if name == "swap":
                a, b = w[:, 0, :, 1], w[:, 1, :, 0]
            elif name == "cx":
                c_hi = qs[0] == hi
                a = w[:, 1, :, 0] if c_hi else w[:, 0, :, 1]
                b = w[:, 1, :, 1]
            else:
                w[:, 1, :, 1] *= -1.0 if name == "cz" else complex(math.cos(ps[0]), math.sin(ps[0]))
                continue
            t = a.clone()
            a.copy_(b)
            b.copy_(t)
            continue
        m = _matrix(name, ps)
        w = v.view(1 << (n - 1 - qs[0]), 2, 1 << qs[0])
        if m[0][1] == 0 and m[1][0] == 0:
            for k in (0, 1):
                if m[k][k] != 1:
                    w[:, k] *= m[k][k]
            continue
        a, b = w[:, 0].clone(), w[:, 1].clone()
        w[:, 0] = m[0][0] * a + m[0][1] * b
        w[:, 1] = m[1][0] * a + m[1][1] * b
    return v


def exact(case, seed):
    if case["use"] not in ("run", "circuit"):
        return None
    n = case["n"]
    v = _simulate(n, _gates(case, seed))
    if case["use"] == "run":
        return dict(statevector=v.cpu().numpy(), samples=None)
    p = v.real.square() + v.imag.square()
    del v
    return dict(p1=np.array([float(p.view(-1, 2, 1 << q)[:, 1].sum()) for q in range(n)]), samples=None)
