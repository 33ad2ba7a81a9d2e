"""Sums of squares of the trajectory engine, on the host (no GPU).

tests/mass_harness.cpp runs the sums behind every probability table
(zeno_gb300/csrc/zc_mass.h) against exact ones: one lane's over 2 to 2^18
squares of several kinds within the bound of its roundings, and table entries
of 5- to 20-qubit states, split over lanes as the kernel splits them, no
further off than 256 unfolded sums.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "zeno_gb300", "csrc")


def test_sums_of_squares(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ is missing")
    exe = str(tmp_path / "mass_harness")
    subprocess.run([cxx, "-std=gnu++17", "-O2", "-Wall", "-Werror", "-ffp-contract=off", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "mass_harness.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "ok sums of squares" in r.stdout, r.stdout
