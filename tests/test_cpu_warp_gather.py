"""The queue through which a warp of the tile-list kernels picks its splats has no two
unordered stores to one place: run on the host with the lanes one after another between
two warp barriers, in ascending, descending and random order, it always places the same
indices."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_queue_does_not_depend_on_the_order_of_lanes(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    exe = tmp_path / "warp_gather"
    r = subprocess.run([cxx, "-std=c++17", "-O1", str(ROOT / "tests" / "cpp" / "warp_gather.cpp"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
