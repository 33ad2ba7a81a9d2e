"""The integer f64 product on the host (no GPU): tests/softmul_harness.cpp
compares zeno_gb300/csrc/zc_softmul.h with the hardware product bit for bit
over edge mantissas, the exponent range's ends, zeros and random operands."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zeno_gb300", "csrc")


def test_products(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is missing")
    exe = str(tmp_path / "softmul_harness")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "softmul_harness.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert out.startswith("ok products"), out
