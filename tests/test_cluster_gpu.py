"""Short sorts by one thread-block cluster (cccl_gb300/csrc/cluster_kernels.cuh) against the oracle,
byte for byte: the smallest and the largest sizes, tiles that are full, ragged or empty, digits that
every key shares, partial bit windows, both result buffers and unaligned arrays."""

import numpy as np
import pytest
import torch

import inputs as I
from gpu_util import from_dev, gpu_sort, to_dev

pytestmark = pytest.mark.gpu


def _most(dtype, value):
    """cluster_max_items in sort_policy.h."""
    width = np.dtype(dtype).itemsize + (0 if value is None else np.dtype(value).itemsize)
    return 16 * 1024 * min(8, 48 // width)


TYPES = [
    (np.uint8, np.uint32),
    (np.uint16, None),
    (np.float32, None),
    (np.int32, np.uint64),
    (np.uint64, np.uint32),
    (np.float64, np.uint64),
]


def _keys(dtype, n, rng):
    dt = np.dtype(dtype)
    if dt.kind == "f":
        return I.with_specials(rng.standard_normal(n).astype(dtype), rng, 1 / 64)
    return I.uniform_bits(np.dtype(f"u{dt.itemsize}"), n, rng).view(dtype)


def _check(oracle, k, v, **kw):
    ko, vo = gpu_sort(k, v, **kw)[:2]
    kw.pop("overwrite", None)
    rk, rv = oracle.radix_sort(k, v, threads=8, **kw)
    assert ko.tobytes() == rk.tobytes()
    assert v is None or vo.tobytes() == rv.tobytes()


@pytest.mark.parametrize("dtype,value", TYPES)
@pytest.mark.parametrize("n", [4865, 8191, 8193, 16 * 1024 - 1, 16 * 1024 * 2, 50021, -1, 0, 1])
def test_sizes(oracle, dtype, value, n):
    if n < 2:
        n += _most(dtype, value)
    rng = np.random.default_rng(n)
    k = _keys(dtype, n, rng)
    v = None if value is None else I.index_values(n, value)
    _check(oracle, k, v)
    _check(oracle, k, v, descending=True, overwrite=True)


@pytest.mark.parametrize("window", [(0, 32), (3, 20), (8, 24), (31, 32), (0, 12)])
@pytest.mark.parametrize("overwrite", [False, True])
def test_bit_windows(oracle, window, overwrite):
    n = 20011
    k = I.uniform_bits(np.uint32, n, np.random.default_rng(5))
    _check(oracle, k, I.index_values(n), begin_bit=window[0], end_bit=window[1], overwrite=overwrite)


@pytest.mark.parametrize("mask", [0, 0xFF, 0xFF00, 0xFF0000FF, 0xFFFFFF00])
def test_shared_digits(oracle, mask):
    n = 30011
    k = I.uniform_bits(np.uint32, n, np.random.default_rng(6)) & np.uint32(mask) | np.uint32(0x5A5A5A5A & ~mask)
    _check(oracle, k, I.index_values(n))
    _check(oracle, np.sort(k), I.index_values(n), descending=True)


def test_unaligned_arrays(oracle):
    from cccl_gb300 import SortOrder, make_radix_sort

    n = 9001
    k = I.uniform_bits(np.uint32, n + 1, np.random.default_rng(7))
    ki, ko = to_dev(k), torch.zeros_like(to_dev(k))
    vi = torch.arange(n + 1, dtype=torch.int32, device="cuda")
    vo = torch.zeros_like(vi)
    args = dict(d_in_keys=ki[1:], d_out_keys=ko[1:], d_in_values=vi[1:], d_out_values=vo[1:])
    s = make_radix_sort(order=SortOrder.ASCENDING, **args)
    temp = torch.empty(s(temp_storage=None, num_items=n, **args), dtype=torch.uint8, device="cuda")
    s(temp_storage=temp, num_items=n, **args)
    rk, rv = oracle.radix_sort(k[1:], np.arange(1, n + 1, dtype=np.int32), threads=8)
    assert from_dev(ko[1:].clone(), np.uint32).tobytes() == rk.tobytes()
    assert from_dev(vo[1:].clone(), np.int32).tobytes() == rv.tobytes()
    assert int(ko[0]) == 0 and int(vo[0]) == 0
