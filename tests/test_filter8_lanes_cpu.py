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
