"""The block fixed-point collision and velocity of the FP64 form
(hemocell_gb300/csrc/hc_blockfixed.h), compiled for the host: over ten decades of
velocity and six of force no further from long double than double arithmetic, and
refused where its bounds do not hold."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_collision_no_further_off_than_double(tmp_path):
    exe = str(tmp_path / "blockfixed_check")
    src = os.path.join(ROOT, "tests", "blockfixed_check.cpp")
    inc = os.path.join(ROOT, "hemocell_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", inc, src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("ok")
