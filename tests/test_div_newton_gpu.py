"""div_newton's proof takes a seed of the reciprocal within 2^-19 (relative):
the hardware's, over every upper word of a divisor and at scales over the range
it is used in, and the quotients formed from it."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_seed_error_and_quotients(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "div_newton_device_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-fmad=false", "-I" + os.path.join(ROOT, "astrosimgpu_b200", "csrc"),
                    os.path.join(ROOT, "tests", "div_newton_device_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    worst, cases, bad = out.split()
    assert float(worst) <= 2.0 ** -19, worst
    assert int(cases) > 30_000_000 and int(bad) == 0, out
