"""Shared-memory limits of the plain sort's kernels on the CPU: radix_sort_dispatch
(cccl_gb300/csrc/radix_plan.cpp) against a driver that records them (tests/host/smem_limit_check.cpp).
Every call has to set the same limit, whatever its size: threads share a build's kernels."""

import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA_INCLUDE = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"


@pytest.mark.skipif(shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda.h").exists(), reason="needs g++ and cuda.h")
def test_limits_do_not_follow_the_size(tmp_path):
    exe = tmp_path / "smem_limit_check"
    csrc = ROOT / "cccl_gb300" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(csrc), "-I", str(ROOT / "include"), "-I",
                    str(CUDA_INCLUDE), str(ROOT / "tests" / "host" / "smem_limit_check.cpp"),
                    str(csrc / "radix_plan.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert "192 sorts, 0 failures" in r.stdout, r.stdout
