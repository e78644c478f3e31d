"""A launch of several steps lists a cell once per step it spikes in; the list
counts records in 28 bits (24 in the latency form) and edges in 32.  span_that_fits
(astrosimgpu_b200/csrc/asg_span.hpp) shortens the launch so that both hold
for a network whose every cell fires as often as its refractory time allows,
whatever the phase: compared with a count over the substeps."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# want, neurons, edges, substeps, refractory substeps
SIZES = [(8, (1 << 25) - 1, 100, 1, 0), (8, 1 << 25, 100, 1, 0), (5, 53_687_091, 100, 1, 0),
         (5, 53_687_092, 100, 1, 0), (8, (1 << 27) - 1, 100, 1, 7), (8, (1 << 27) - 1, 100, 1, 6),
         (8, 1 << 28, 100, 1, 20), (5, 10, 845_571_686, 1, 0), (5, 10, 845_571_687, 1, 0),
         (8, 1000, (1 << 32) - (1 << 26), 1, 20), (8, 1000, (1 << 32) - (1 << 26) + 1, 1, 20),
         (8, 4_000_000, 400_000_000, 2, 5), (8, 8_000_000, 900_000_000, 1, 3),
         (8, 96_000_000, 10, 3, 2), (4, 80_000_000, 10, 1, 1), (1, 1 << 24, 1 << 33, 1, 0),
         (8, 500, 25_000, 1, 20), (5, 1_000_000, 10**8, 1, 0), (8, 0, 0, 1, 0)]
CASES = [c + (28,) for c in SIZES] + [(c[0], c[1] >> 4) + c[2:] + (24,) for c in SIZES]


@pytest.fixture(scope="module")
def limits(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path_factory.mktemp("spanlimit") / "span_limit_check")
    subprocess.run([cxx, "-std=c++17", "-I" + os.path.join(ROOT, "astrosimgpu_b200", "csrc"),
                    os.path.join(ROOT, "tests", "span_limit_check.cpp"), "-o", exe], check=True)
    text = "\n".join(" ".join(map(str, c)) for c in CASES)
    out = subprocess.run([exe], input=text, check=True, capture_output=True, text=True).stdout
    return [list(map(int, line.split())) for line in out.splitlines()]


def counted(steps, substeps, ref):
    """Most steps with a spike in any window of `steps`, the cell firing in
    every substep it may."""
    most = 0
    for phase in range(ref + 1):
        hit = {k // substeps for k in range(phase, steps * substeps, ref + 1)}
        most = max(most, len(hit))
    return most


@pytest.mark.parametrize("k", range(len(CASES)))
def test_spikes_of_a_launch_fit_its_list(limits, k):
    want, n, e, substeps, ref, bits = CASES[k]
    span, *spikes = limits[k]
    assert spikes == [counted(L, substeps, ref) for L in range(1, want + 1)]

    def fits(L):
        s = counted(L, substeps, ref)
        return s * n < 1 << bits and s * e + (1 << 26) <= 1 << 32

    assert span == max([1] + [L for L in range(2, want + 1) if fits(L)])

