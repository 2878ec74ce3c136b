"""Kernels opt in to large shared memory once per device, not once per process: with a fake
of the runtime's two calls, and no other place in the sources that sets the attribute."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_opt_in_is_per_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cxx, inc = shutil.which("g++"), Path(nvcc).resolve().parents[1] / "include"
    if not cxx or not (inc / "cuda_runtime_api.h").exists():
        pytest.skip("no host compiler or CUDA headers")
    exe = tmp_path / "smem_optin"
    r = subprocess.run([cxx, "-std=c++17", "-I", str(inc),
                        str(ROOT / "tests" / "cpp" / "smem_optin.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def test_every_kernel_opts_in_through_the_helper():
    for f in sorted((ROOT / "diffsplat_b200" / "csrc").iterdir()):
        if f.name != "ds_smem.h":
            assert "MaxDynamicSharedMemorySize" not in f.read_text(), f.name
