"""The lanes of a warp may run in any order between two warp-wide operations: the traversals by groups of eight lanes,
compiled for the host, give the results of one thread per ray whatever order their lanes take."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_group_traversal_does_not_depend_on_the_lane_order(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = tmp_path / "warp_lanes"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-ffp-contract=off", "-w", "-I/usr/local/cuda/include",
                        str(ROOT / "tests" / "cxx" / "warp_lanes.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
