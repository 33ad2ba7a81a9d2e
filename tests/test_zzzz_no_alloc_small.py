"""Sampling without allocation from a small state whose gates still wait.

A state under 14 qubits launches its waiting ops inside zc_sample_noalloc, and
loading a kernel can allocate device memory. In a fresh process each, with
only the sampler's own kernels loaded before, the call leaves the device's
free memory alone whatever the ops; a state created with the forcing flag is
refused until zc_finish, as are larger ones.
"""

import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys
import numpy as np
from zeno_gb300 import backend as zc
prec, flags, what = int(sys.argv[1]), int(sys.argv[2]), sys.argv[3]
cu = ctypes.CDLL("libcuda.so.1")
def free():
    a, b = ctypes.c_size_t(), ctypes.c_size_t()
    assert cu.cuMemGetInfo_v2(ctypes.byref(a), ctypes.byref(b)) == 0
    return a.value
warm = zc.CudaBackend(12, prec, flags)
warm.sample_noalloc(64, 1)
be = zc.CudaBackend(9, prec, flags)
be.finish()
h = np.array([[1, 1], [1, -1]]) / np.sqrt(2)
def dense(k):
    m = np.eye(1 << k, dtype=complex)
    m[-2:, -2:] = h
    be.apply_unitary(list(range(9 - k, 9)), m)
def gates(count):
    for i in range(count):
        be.apply_unitary([i % 9], h)
        be.apply_cx(i % 9, (i + 4) % 9)
        be.apply_diagonal([i % 9, 8] if i % 9 < 8 else [8], np.exp(1j * np.arange(4 if i % 9 < 8 else 2)))
if what == "few":
    gates(1)
elif what == "many":
    gates(40)
else:
    gates(20)
    for k in range(2, 8):
        dense(k)
        gates(5)
f0 = free()
got = be.sample_noalloc(1000, 3)
f1 = free()
assert f0 == f1, (f0, f1)
exact = zc.CudaBackend(9, prec, zc.FLAG_EXACT)
exact.load_state(be.statevector())
assert np.array_equal(got, exact.sample(1000, 3))
print("nothing allocated")
"""


@pytest.mark.parametrize("what", ("few", "many", "dense"))
@pytest.mark.parametrize("prec,flags", ((64, 0), (64, 1), (32, 1), (32, 17)))
def test_waiting_gates_allocate_nothing(zc, prec, flags, what):
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(prec), str(flags), what], cwd=ROOT, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0 and "nothing allocated" in r.stdout, r.stderr


def test_forced_sweeps_are_refused_until_finish(zc):
    be = zc.CudaBackend(8, 64, zc.FLAG_FORCE_SWEEPS)
    be.apply_cx(0, 1)
    with pytest.raises(zc.ZenoCudaError, match="zc_finish"):
        be.sample_noalloc(10, 1)
    be.finish()
    assert np.array_equal(be.sample_noalloc(10, 1), np.zeros(10))
    be.close()
