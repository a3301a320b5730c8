"""The scatter term's quick polar range against the reference-order one, on the host
(csrc/scatter_term.cuh is host-callable): the number of 0.01 rad steps, which decides
terms of the Klein-Nishina sum, is the same always, the angles within 5e-7 rad (the
quick form's 3e-7 and the exact one's rounding at up to pi)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("polar") / "check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I/usr/local/cuda/include",
                           "-I" + os.path.join(ROOT, "gpu-spect-pet-sysmat_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                           os.path.join(HERE, "polar_range_check.cpp"), "-o", exe])
    return exe


@pytest.mark.parametrize("distance", [4, 20, 90])
def test_step_counts_are_the_exact_ones(check, distance):
    n, other, lo_diff, angle_err = subprocess.check_output([check, "3", "400000", str(distance)], text=True).split()
    assert int(other) == 0, (n, other)
    assert float(lo_diff) <= 5e-7 and float(angle_err) <= 4e-7
