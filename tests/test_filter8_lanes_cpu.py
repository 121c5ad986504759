"""The 8-lane collaborative filter (csrc/zb3d_filter.cuh) on the CPU, its lanes as fibers that
change only at warp-wide operations (tests/lanes): an order the hardware may take, in which a
value read after another lane has replaced it gives a wrong sum."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "vapoursynth-zipcu_b200", "csrc")


@pytest.fixture(scope="module")
def filter8(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("lanes") / "filter8")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-I", os.path.join(HERE, "lanes"),
                           "-I", CSRC, os.path.join(HERE, "lanes", "filter8.cpp"), "-o", exe])
    return exe


@pytest.mark.parametrize("final", [0, 1])
@pytest.mark.parametrize("descending", [0, 1])
def test_groups_after_groups_in_the_same_buffers(filter8, final, descending):
    assert subprocess.run([filter8, "chunk", str(final), str(descending)]).returncode == 0


@pytest.mark.parametrize("final", [0, 1])
@pytest.mark.parametrize("exponent,rounds_to_zero", [(3, False), (95, True), (96, True), (100, True), (127, True)])
def test_extractor_exponents(filter8, final, exponent, rounds_to_zero):
    """v + 2^e - 2^e: the spacing of floats at 2^e is 2^(e - 23), so with e from 26 up every weighted pixel and weight of [0, 1] data rounds to
    zero, also where 2^e scaled to the accumulators' fixed point would be infinite."""
    counts = list(map(int, subprocess.check_output([filter8, "sums", str(final), str(exponent)]).split()))
    assert (counts == [0, 0]) == rounds_to_zero, counts
