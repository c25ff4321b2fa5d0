"""The voxelizer's host side on a CUDA runtime that the test makes itself (fake_cuda_vox.cpp). A call that fails after its
upload was queued waits for it: the pinned tables and the scratch belong to the next call, and the caller's models to the
caller. The order of mixed lists holds, and costs little where few ops differ."""
import os
import shutil
import subprocess

import pytest

from voxelengine_gb300 import buildlib

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    exe = tmp_path_factory.mktemp("fake") / "fake"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(buildlib.nvcc()))), "include")
    # the launches that these calls do not reach stay unresolved
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-I", cuda, "-I", buildlib.INCLUDE, "-I",
                    buildlib.CSRC, os.path.join(HERE, "fake_cuda_vox.cpp"), os.path.join(buildlib.CSRC, "vxl_api.cpp"),
                    "-o", str(exe), "-Wl,--unresolved-symbols=ignore-all"], check=True)
    return lambda *args: subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, check=True,
                                        timeout=120).stdout


def test_failing_calls_leave_nothing_queued(fake):
    rows = [tuple(map(int, line.split())) for line in fake().splitlines()]
    # level, read-back, event, tile mask and wait fail in turn, after a call where nothing does
    assert [r[0] for r in rows] == [0, 1, 2, 3, 4, 5]
    assert [r[1] != 0 for r in rows] == [False, True, True, True, True, True]
    assert [r[2] for r in rows] == [0] * 6


@pytest.mark.parametrize("what", ["one", "halves", "pairs", "third"])
@pytest.mark.parametrize("n", [1, 2, 7, 600, 1500, 6000])
def test_order_of_mixed_lists(fake, what, n):
    levels = int(fake(what, n).split()[0])
    assert 1 <= levels <= n


def test_few_differing_ops_cost_little(fake):
    """A test of every pair of a segment of 1,024 took 55 ms for these, most of it on pairs of one op."""
    for what in ("one", "halves"):
        levels, ms = fake(what, 65536).split()
        assert float(ms) < 20.0
        assert int(levels) <= 4
