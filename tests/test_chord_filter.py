"""The tracer's chord filters (boxes, holes) against the reference-order chords, on
the host: the same header (csrc/tracer.cuh) the kernels include.  The filter may
call a chord unclear, never wrong; a clear chord lies within the filter's own
margin of the exact one (both ends of the chord move by less than the margin
times the ray's slope)."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gpu-spect-pet-sysmat_b200", "csrc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("chord") / "check")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I/usr/local/cuda/include", "-I" + CSRC,
                           os.path.join(HERE, "chord_filter_check.cpp"), "-o", exe])
    return exe


@pytest.mark.parametrize("coordinate_range", [20, 128, 700])
def test_clear_calls_are_the_exact_ones(check, coordinate_range):
    out = subprocess.check_output([check, "5", "1500000", str(coordinate_range)], text=True).split()
    wrong, hits, misses, unclear = map(int, out[:4])
    assert wrong == 0, out
    assert hits > 100000 and misses > 100000
    assert unclear < 0.35 * (hits + misses)      # every second ray aims at an edge
    assert float(out[4]) <= 2.0
    hole_misses, hole_hits, hole_other, other, flat = map(int, out[5:])
    assert hole_misses > 50000 and hole_hits > 50000        # three holes in five have their wall near the ray
    assert other < 1e-2 * hits and flat > 10000
    assert hole_other < 1e-3 * hole_hits                    # the exact form's value but for rare last bits
