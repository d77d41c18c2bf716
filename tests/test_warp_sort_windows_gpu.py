"""Bit windows of 4-byte keys in segments that one warp sorts (cccl_gb300/csrc/warp_sort.cuh): around the
widths at which its elements change from 32 to 64 bits, against the oracle, byte for byte."""

import numpy as np
import pytest

import inputs as I
from gpu_util import gpu_seg_sort
from segments import edge_segments

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,value", [(np.uint32, None), (np.int32, np.uint64), (np.float32, np.uint32)])
@pytest.mark.parametrize("window", [(0, 1), (0, 8), (5, 21), (16, 32), (15, 32), (4, 21), (1, 32)])
def test_widths(oracle, dtype, value, window):
    rng = np.random.default_rng(23)
    b, e, n = edge_segments([257, 258, 300, 384, 385, 511, 512] * 20, gap=3)
    k = I.uniform_bits(np.uint32, n, rng)
    k[rng.random(n) < 0.1] |= np.uint32(0xFFFFFFFF >> 4)  # windows of all ones, next to the padding
    k = k.view(dtype)
    if np.dtype(dtype).kind == "f":
        k[np.isnan(k)] = 1.5
    v = None if value is None else I.index_values(n, value)
    for desc, overwrite in ((False, False), (True, True)):
        ko, vo, _ = gpu_seg_sort(k, v, b, e, descending=desc, overwrite=overwrite, radix_bits=window)
        for lo, hi in zip(b, e):
            rk, rv = oracle.radix_sort(k[lo:hi], None if v is None else v[lo:hi], window[0], window[1], desc, threads=1)
            assert ko[lo:hi].tobytes() == rk.tobytes()
            assert v is None or vo[lo:hi].tobytes() == rv.tobytes()
