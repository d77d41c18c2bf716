"""Shared memory of the segmented sort's block classes (cccl_gb300/csrc/sort_policy.h), for the
default block algorithm and for the merge sort that tuning builds select
(tests/host/block_smem_check.cpp, compiled with g++)."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("defines", [[], ["-DGB300_SEG_BLOCK_ALGO=1"], ["-DGB300_SEG_BLOCK_ALGO=1", "-DGB300_SEG_BLOCK_L_ITEMS=8"]])
def test_every_form_fits(tmp_path, defines):
    exe = tmp_path / "block_smem_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", *defines, "-I", str(ROOT / "cccl_gb300" / "csrc"),
                    str(ROOT / "tests" / "host" / "block_smem_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
