"""The block fixed-point collision of the FP64 form over every relaxation time that
a handle accepts, compiled for the host, against long double."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_relaxation_times(tmp_path):
    exe = str(tmp_path / "relaxation_check")
    src = os.path.join(ROOT, "tests", "relaxation_check.cpp")
    inc = os.path.join(ROOT, "hemocell_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", inc, src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("ok")
