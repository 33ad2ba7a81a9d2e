"""The op queue of a state or request, on the host (no GPU).

tests/queue_harness.cpp walks queues of random ops (dense blocks among them,
up to 5000 ops) from their head and, beside that, as a vector whose front is
taken out: every plan is the same. Then it times the walk over dense blocks
and CX in turn: the host time per op is that of a short queue however long the
queue is (it grew thirtyfold to 8000 ops when each op's removal moved the rest).
"""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zeno_gb300", "csrc")


def test_queue_plans_and_cost(zc, tmp_path):
    from zeno_gb300 import build

    cxx = shutil.which("g++")
    inc = next((os.path.join(b, "include") for b in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                if b and os.path.exists(os.path.join(b, "include", "cuda_runtime.h"))), None)
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path / "queue_harness")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I" + CSRC, "-I" + inc,
                    os.path.join(ROOT, "tests", "queue_harness.cpp"), build.LIB,
                    "-Wl,-rpath," + os.path.dirname(build.LIB), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    m = re.match(r"ok plans; host us per op: (\S+) of 250 ops, (\S+) of 8000", r.stdout)
    assert r.returncode == 0 and m, r.stdout
    assert float(m[2]) < 3.0 * float(m[1]), r.stdout
