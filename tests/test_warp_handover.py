"""Warps hand slots back by one lane's arrive.  Every lane has to be past its own wait on the slot by then: the arrive
lets the slot be filled again, and a lane that still polls the old phase's parity would miss it.  No run shows a missing
barrier reliably, so the sources are read."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "tritium_b200", "csrc")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "kernels_*.cu"))), ids=os.path.basename)
def test_a_lane_arrives_for_its_warp_behind_a_warp_barrier(path):
    code = [re.sub(r"//.*", "", line).strip() for line in open(path)]
    code = [line for line in code if line]
    for i, line in enumerate(code):
        if line.startswith("if (lane == 0) mbar_arrive("):
            assert code[i - 1] == "__syncwarp();", f"{os.path.basename(path)}: {line}"
