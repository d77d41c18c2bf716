"""Plain sorts whose output is their input. The route is checked on the CPU, radix_sort_dispatch
(cccl_gb300/csrc/radix_plan.cpp) against a recording driver (tests/host/in_place_check.cpp), the
result on the GPU."""

import os
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import inputs as I

ROOT = Path(__file__).resolve().parent.parent
CUDA_INCLUDE = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"


@pytest.mark.skipif(shutil.which("g++") is None or not (CUDA_INCLUDE / "cuda.h").exists(), reason="needs g++ and cuda.h")
def test_every_pass_runs(tmp_path):
    exe = tmp_path / "in_place_check"
    csrc = ROOT / "cccl_gb300" / "csrc"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(csrc), "-I", str(ROOT / "include"), "-I",
                    str(CUDA_INCLUDE), str(ROOT / "tests" / "host" / "in_place_check.cpp"),
                    str(csrc / "radix_plan.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_result(oracle):
    """Normal doubles, which the sort into another buffer partitions by three digits."""
    import torch

    from cccl_gb300 import SortOrder, make_radix_sort
    from gpu_util import from_dev, to_dev

    n = 5_000_003
    keys = np.random.default_rng(29).standard_normal(n)
    k, v = to_dev(keys), to_dev(I.index_values(n))
    args = dict(d_in_keys=k, d_out_keys=k, d_in_values=v, d_out_values=v)
    s = make_radix_sort(order=SortOrder.ASCENDING, **args)
    temp = torch.empty(s(temp_storage=None, num_items=n, **args), dtype=torch.uint8, device="cuda")
    s(temp_storage=temp, num_items=n, **args)
    rk, rv = oracle.radix_sort(keys, I.index_values(n), threads=8)
    assert from_dev(k, np.float64).tobytes() == rk.tobytes()
    assert from_dev(v, np.uint32).tobytes() == rv.tobytes()
