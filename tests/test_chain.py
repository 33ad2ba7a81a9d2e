"""Serial f64 sums evaluated in parallel, on the host (no GPU).

tests/chain_harness.cpp reduces rows of 32 values with the functions the
reduction kernels use (zeno_gb300/csrc/zc_chain.h) and compares every row's
start and the result with plain serial additions, bit for bit: f64 and f32
amplitude masses, ties, powers of two, sparse, uniform, subnormal, infinite
and NaN values, from several starting sums.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zeno_gb300", "csrc")


def test_serial_sums_in_parallel(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is missing")
    exe = str(tmp_path / "chain_harness")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-ffp-contract=off", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "chain_harness.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert out.startswith("ok chains"), out
