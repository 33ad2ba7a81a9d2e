"""Sweep jobs with operands out of range are refused on the host (no GPU).

tests/operands_harness.cpp encodes one-op jobs through the built library's own
encode_job, for every arithmetic and kind of op, with operands at the last
place inside the tile, the state and the tables and at the first outside.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zeno_gb300", "csrc")


def test_operands_are_checked(zc, tmp_path):
    from zeno_gb300 import build

    cxx = shutil.which("g++")
    inc = next((os.path.join(b, "include") for b in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                if b and os.path.exists(os.path.join(b, "include", "cuda_runtime.h"))), None)
    if cxx is None or inc is None:
        pytest.skip("g++ or the CUDA headers are missing")
    exe = str(tmp_path / "operands_harness")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I" + CSRC, "-I" + inc,
                    os.path.join(ROOT, "tests", "operands_harness.cpp"), build.LIB,
                    "-Wl,-rpath," + os.path.dirname(build.LIB), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok operands"), r.stdout
