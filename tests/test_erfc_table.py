"""The scatter term's tabulated erfc on the host (csrc/scatter_term.cuh is host-callable):
within half a unit of the stored value and half a unit of the result (2 x 6e-8 of erfc,
1.25e-7 with the slope's rounding), plus the cubic's remainder and the cut at +-4.25 (3e-9)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("erfc") / "check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I/usr/local/cuda/include",
                           "-I" + os.path.join(ROOT, "gpu-spect-pet-sysmat_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                           os.path.join(HERE, "erfc_table_check.cpp"), "-o", exe])
    return exe


@pytest.mark.parametrize("low,high", [(-1.5, 1.5), (1.4, 4.3), (-4.3, -1.4), (-20, 20)])
def test_error_is_rounding(check, low, high):
    worst = float(subprocess.check_output([check, "7", "400000", str(low), str(high)], text=True))
    assert worst <= 1.0
