"""The scatter term's tabulated window probability on the host (csrc/scatter_term.cuh is
host-callable), for wide windows and narrow ones.  One that holds E' is a multiple of the sum
of two erf: half a unit each of erf, of the sum and of the product, 1.8e-7 of it, with 2e-8
for the cubic's remainder and its small terms.  One beside E' is half the difference of two
erfc, each within half a unit of the larger (6e-8 and as much for their difference) and the
3e-9 cut off at the table's end."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("window") / "check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I/usr/local/cuda/include",
                           "-I" + os.path.join(ROOT, "gpu-spect-pet-sysmat_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                           os.path.join(HERE, "window_probability_check.cpp"), "-o", exe])
    return exe


@pytest.mark.parametrize("width", [2.0, 0.5, 0.1, 0.02, 0.005, 0.0002])
def test_narrow_windows_lose_nothing(check, width):
    across, beside = map(float, subprocess.check_output([check, "11", "400000", str(width)], text=True).split())
    assert across <= 2.0e-7 and beside <= 1.3e-7
