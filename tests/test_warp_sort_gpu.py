"""Segments sorted in the registers of one warp or of a group of warps (cccl_gb300/csrc/warp_sort.cuh):
lengths around every change of the form, ragged starts, shared digits, partial bit windows and one
buffer for input and output, against the oracle, byte for byte."""

import numpy as np
import pytest

import inputs as I
from gpu_util import gpu_seg_sort
from segments import edge_segments

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 18, 19, 31, 32, 33, 57, 63, 64, 65, 112, 113, 127, 128, 129, 255, 256, 257, 300, 511, 512, 513]
LENGTHS += [700, 1023, 1024, 1025, 1500, 2047, 2048, 2049]
TYPES = [
    (np.int32, None),
    (np.uint32, None),
    (np.uint16, None),
    (np.uint8, np.uint32),
    (np.float16, np.uint32),
    (np.float32, None),
    (np.float32, np.uint32),
    (np.int32, np.uint64),
]


def _keys(dtype, n, rng, spread):
    dt = np.dtype(dtype)
    if dt.kind == "f":
        k = rng.standard_normal(n).astype(dtype)
        return k if spread else I.with_specials(k, rng, 0.3)
    k = I.uniform_bits(np.dtype(f"u{dt.itemsize}"), n, rng)
    if not spread:  # few keys, the largest and the smallest among them
        k = np.array([0, 1, 2, ~np.uint64(0), ~np.uint64(0) >> np.uint64(1)], np.uint64).astype(k.dtype)[rng.integers(0, 5, n)]
    return k.view(dtype)


@pytest.mark.parametrize("dtype,value", TYPES)
@pytest.mark.parametrize("spread", [True, False])
@pytest.mark.parametrize("bits", [None, (0, None), (3, 7)])
def test_lengths(oracle, dtype, value, spread, bits):
    rng = np.random.default_rng(21)
    b, e, n = edge_segments(LENGTHS * 40, gap=5)
    k = _keys(dtype, n, rng, spread)
    v = None if value is None else I.index_values(n, value)
    for desc, overwrite in ((False, False), (True, True)):
        if bits is None:
            rk, rv = oracle.segmented_sort(k, v, b, e, descending=desc, threads=8)
        else:
            rk, rv = k.copy(), None if v is None else v.copy()
            for lo, hi in zip(b, e):
                sk, sv = oracle.radix_sort(k[lo:hi], None if v is None else v[lo:hi], bits[0], bits[1], desc, threads=1)
                rk[lo:hi] = sk
                if v is not None:
                    rv[lo:hi] = sv
        ko, vo, _ = gpu_seg_sort(k, v, b, e, descending=desc, overwrite=overwrite, radix_bits=bits)
        ok = np.zeros(n, bool)
        for lo, hi in zip(b, e):
            ok[lo:hi] = True
        assert ko[ok].tobytes() == rk[ok].tobytes()
        assert v is None or vo[ok].tobytes() == rv[ok].tobytes()


def test_few_segments(oracle):
    """Too few segments to split the short ones into classes."""
    b, e, n = edge_segments([1, 3, 17, 33, 100, 200, 400, 2000, 3000], gap=3)
    k = I.uniform_bits(np.uint32, n, np.random.default_rng(22))
    rk, _ = oracle.segmented_sort(k, None, b, e, descending=False, threads=8)
    ko, _, _ = gpu_seg_sort(k, None, b, e)
    for lo, hi in zip(b, e):
        assert ko[lo:hi].tobytes() == rk[lo:hi].tobytes()
