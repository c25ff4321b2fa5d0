"""A voxelizer call that fails after its upload was queued waits for it: the pinned tables and the scratch belong to the
next call, and the caller's models to the caller. Host code only, on a CUDA runtime that the test makes itself."""
import os
import shutil
import subprocess

import pytest

from voxelengine_gb300 import buildlib

HERE = os.path.dirname(os.path.abspath(__file__))


def test_failing_calls_leave_nothing_queued(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    exe = tmp_path / "fake"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(buildlib.nvcc()))), "include")
    # the launches that this call does not reach stay unresolved
    subprocess.run([cxx, "-std=c++17", "-O1", "-w", "-I", cuda, "-I", buildlib.INCLUDE, "-I", buildlib.CSRC,
                    os.path.join(HERE, "fake_cuda_vox.cpp"), os.path.join(buildlib.CSRC, "vxl_api.cpp"), "-o", str(exe),
                    "-Wl,--unresolved-symbols=ignore-all"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=60).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    # level, read-back, event, tile mask and wait fail in turn, after a call where nothing does
    assert [r[0] for r in rows] == [0, 1, 2, 3, 4, 5]
    assert [r[1] != 0 for r in rows] == [False, True, True, True, True, True]
    assert [r[2] for r in rows] == [0] * 6
