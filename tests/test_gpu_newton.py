"""hcnewton::recip and inv_length on the device, from the hardware's approximate
seeds: within 2^-52 of 1/x, 1/sqrt(x) and sqrt(x), the bound that their seed
accuracy gives (hemocell_gb300/csrc/hc_newton.h), over all binades."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reciprocals_on_the_device(built, tmp_path):
    from hemocell_gb300 import build as b
    exe = str(tmp_path / "newton_gpu_check")
    subprocess.run([b._nvcc(), b.GENCODE, "-O3", "-std=c++17", "-I", b.CSRC, "-o", exe,
                    os.path.join(ROOT, "tests", "newton_gpu_check.cu")], check=True, capture_output=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().splitlines()[-1].startswith("ok ")
