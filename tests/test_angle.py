"""The scatter term's angle_quick on the host (csrc/scatter_term.cuh is host-callable)
against atan2 in double.  The reduced angle: its polynomial's 2.3e-8, half a unit of the
quotient and of the result (6e-8 each) and a fifth of a unit of the polynomial's rounding,
1.6e-7 of it, 1.3e-7 at pi / 4.  Beyond, half a unit of a number below 0.8 (3e-8) and of the
result are added: 6e-8 up to pi / 2, 1.2e-7 up to pi."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.parametrize("seed", [1, 2])
def test_error_is_rounding(tmp_path, seed):
    exe = str(tmp_path / "check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I/usr/local/cuda/include",
                           "-I" + os.path.join(ROOT, "gpu-spect-pet-sysmat_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                           os.path.join(HERE, "angle_check.cpp"), "-o", exe])
    low, mid, high, axes = map(float, subprocess.check_output([exe, str(seed), "2000000"], text=True).split())
    assert low <= 1.6e-7 and mid <= 2.2e-7 and high <= 2.8e-7 and axes == 1
