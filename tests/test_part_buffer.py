"""A failed allocation of the partial sums' buffer leaves no capacity behind, on
the host (no GPU): tests/part_harness.cpp asks for sums of a state of 2^58
amplitudes, whose buffer no machine can give."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zeno_gb300", "csrc")


def test_failed_allocation_leaves_no_capacity(zc, tmp_path):
    from zeno_gb300 import build

    cxx = shutil.which("g++")
    inc = next((os.path.join(b, "include") for b in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                if b and os.path.exists(os.path.join(b, "include", "cuda_runtime.h"))), None)
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path / "part_harness")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I" + CSRC, "-I" + inc,
                    os.path.join(ROOT, "tests", "part_harness.cpp"), build.LIB,
                    "-Wl,-rpath," + os.path.dirname(build.LIB), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout
