"""Whole runs of the block fixed-point collision of the FP64 form (walls, an obstacle,
periodic, several relaxation times), compiled for the host: no further from long
double than double arithmetic in any set-up."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_runs_no_further_off_than_double(tmp_path):
    exe = str(tmp_path / "lattice_error_check")
    src = os.path.join(ROOT, "tests", "lattice_error_check.cpp")
    inc = os.path.join(ROOT, "hemocell_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", inc, src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
