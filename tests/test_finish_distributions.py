"""The plain sort's choice for samples of known distributions (finish_choose in cccl_gb300/csrc/sort_policy.h), compiled with
g++ (tests/host/finish_distributions_check.cpp)."""

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_distributions(tmp_path):
    exe = tmp_path / "finish_distributions_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(ROOT / "cccl_gb300" / "csrc"),
                    str(ROOT / "tests" / "host" / "finish_distributions_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
