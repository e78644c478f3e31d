"""div_newton, the engine's division by a divisor computed on the fly
(astrosimgpu_b200/csrc/asg_device.cuh), is bitwise the IEEE quotient for every
divisor it is used on and any seed within its error bound:
tests/div_newton_check.cu runs it on the host over random operands, the whole
exponent range it is used in, divisors at the edges (next to the excluded
ones, next to one, few bits set), quotients as close to a midpoint of two
doubles as 53-bit operands allow, and the operands of the astrocyte model."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("divnewton") / "div_newton_check")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-x", "cu", "-Wno-deprecated-gpu-targets",
                    "-Xcompiler", "-ffp-contract=off",
                    "-I" + os.path.join(ROOT, "astrosimgpu_b200", "csrc"),
                    os.path.join(ROOT, "tests", "div_newton_check.cu"), "-o", exe],
                   check=True, capture_output=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_div_newton_equals_ieee_division(checker, seed):
    out = subprocess.run([checker, "10000000", str(seed)], check=True, capture_output=True,
                         text=True)
    rows = {name: (int(cases), int(bad))
            for name, cases, bad in (line.split() for line in out.stdout.splitlines())}
    assert set(rows) == {"random", "wide", "edge", "midpoint", "model"}
    for name, (cases, bad) in rows.items():
        assert cases > 1_000_000, (name, cases)
        assert bad == 0, (name, cases, bad, out.stderr[:500])
