"""Segmented sorts back to back on one stream and one temporary storage, with a kernel in between that
rewrites the keys and the segments' bounds: the class kernels start before the launches in front of
them have ended (chain_begin in cccl_gb300/csrc/sort_common.cuh) and must see this call's segments."""

import numpy as np
import pytest
import torch

import inputs as I
from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu

ROUNDS = 8


def _bounds(rng, n, shape):
    """Bounds of as many segments as every round has, over the n keys: every class of lengths in turn."""
    nseg = 700
    if shape % 4 == 0:  # short ones, the rest in one long segment
        length = rng.integers(0, 300, nseg)
    elif shape % 4 == 1:  # 100 to 2000
        length = rng.integers(100, 2000, nseg)
    elif shape % 4 == 2:  # a few long ones among empty ones
        length = np.where(rng.random(nseg) < 0.03, rng.integers(4000, 40000, nseg), 0)
    else:
        length = np.exp(rng.normal(5.0, 2.0, nseg)).astype(np.int64)
    ends = np.minimum(np.cumsum(length), n)
    ends[-1] = n
    return np.concatenate([[0], ends]).astype(np.int32)


@pytest.mark.parametrize("key,value", [(np.int32, None), (np.float32, np.int32), (np.float64, np.int64)])
@pytest.mark.parametrize("captured", [False, True])
def test_bounds_rewritten_between_calls(oracle, key, value, captured):
    from cccl_gb300 import SortOrder, make_segmented_sort

    rng = np.random.default_rng(41)
    n = 600_011
    bounds = np.stack([_bounds(rng, n, r) for r in range(ROUNDS)])
    keys = [rng.standard_normal(n).astype(key) if np.dtype(key).kind == "f" else I.uniform_bits(np.uint32, n, rng).view(key)
            for _ in range(ROUNDS)]
    all_bounds = torch.from_numpy(bounds).cuda()
    all_keys = torch.stack([to_dev(k) for k in keys])
    now = torch.zeros(bounds.shape[1], dtype=torch.int32, device="cuda")
    ki = torch.zeros_like(all_keys[0])
    ko = torch.zeros_like(ki)
    vi = None if value is None else to_dev(I.index_values(n, value))
    vo = None if value is None else torch.zeros_like(vi)
    arrays = dict(d_in_keys=ki, d_out_keys=ko, d_in_values=vi, d_out_values=vo)
    offsets = dict(start_offsets_in=now[:-1], end_offsets_in=now[1:])
    s = make_segmented_sort(order=SortOrder.ASCENDING, **arrays, **offsets)
    call = dict(num_items=n, num_segments=bounds.shape[1] - 1, **arrays, **offsets)
    temp = torch.empty(s(temp_storage=None, **call), dtype=torch.uint8, device="cuda")
    out_keys = torch.zeros_like(all_keys)
    out_values = None if value is None else torch.zeros((ROUNDS, n), dtype=vi.dtype, device="cuda")

    def steps():
        for r in range(ROUNDS):
            torch.add(all_bounds[r], 0, out=now)  # kernels, not copies: the sort's first launch follows one
            torch.mul(all_keys[r], 1, out=ki)
            s(temp_storage=temp, **call)
            torch.mul(ko, 1, out=out_keys[r])
            if value is not None:
                torch.add(vo, 0, out=out_values[r])

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        steps()
    side.synchronize()
    if captured:
        out_keys.zero_()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            steps()
        graph.replay()
        graph.replay()
    torch.cuda.synchronize()
    for r in range(ROUNDS):
        v = None if value is None else I.index_values(n, value)
        rk, rv = oracle.segmented_sort(keys[r], v, bounds[r][:-1], bounds[r][1:], threads=8)
        assert from_dev(out_keys[r], key).tobytes() == rk.tobytes()
        if value is not None:
            assert from_dev(out_values[r], value).tobytes() == rv.tobytes()
