"""Votes and reductions of part of a warp name their lanes by an earlier vote of the whole warp: __activemask() gives the
lanes that happen to run together at that point, which need not be those that reach the vote together."""
import os
import re

import pytest

from voxelengine_gb300 import buildlib


@pytest.mark.parametrize("name", ["march_pool.cuh", "trace.cu", "soft.cu", "taa.cu", "primary.cu", "voxelize.cu", "voxel_tile.cuh"])
def test_no_vote_on_the_active_lanes(name):
    text = open(os.path.join(buildlib.CSRC, name)).read()
    assert not re.findall(r"_sync\(\s*__activemask", text)
