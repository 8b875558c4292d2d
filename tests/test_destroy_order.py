"""Destroying a BVH waits for the device that holds it before its memory goes back, with and without a context:
the destroy calls run on the CPU against a recording stand-in for the CUDA runtime with two devices."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_destroy_waits_for_the_trees_device(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = tmp_path / "destroy_order"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-I/usr/local/cuda/include",
                        str(ROOT / "tests" / "cxx" / "destroy_order.cpp"),
                        str(ROOT / "vierkant_gb300" / "csrc" / "destroy.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
