"""Limits of the cycle graph's tile list and of its grids, on the host (tests/tile_list_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "salec-2d-public_b200", "csrc")


def test_tile_entries_and_grids(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++ on this machine")
    exe = str(tmp_path / "tile_list_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", CSRC, "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "tile_list_check.cpp"), "-o", exe], check=True, capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr
