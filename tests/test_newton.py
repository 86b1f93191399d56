"""The FP64 reciprocal, reciprocal square root and integer floor of the cell
kernels (hemocell_gb300/csrc/hc_newton.h, hc_posbits.h), compiled for the host,
against long double and floor()."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_newton_steps_and_floor_bits(tmp_path):
    exe = str(tmp_path / "newton_check")
    src = os.path.join(ROOT, "tests", "newton_check.cpp")
    inc = os.path.join(ROOT, "hemocell_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", inc, src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[1]) == 5_000_000
