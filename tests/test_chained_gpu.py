"""Overlapped launches of short sorts (launch_after in cccl_gb300/csrc/abi_common.h) and the pass with
one tile per CTA (onesweep.cuh): sizes around the last one that has a tile for every CTA, and sorts
directly behind the kernels that write their input and before the ones that read their output."""

import numpy as np
import pytest
import torch

import inputs as I
from gpu_util import from_dev, gpu_sort, to_dev

pytestmark = pytest.mark.gpu

# items of a tile of the persistent pass: main threads * items per thread (sort_policy.h)
TILES = [
    (np.uint32, None, 768 * 14),
    (np.float32, np.uint32, 640 * 13),
    (np.uint64, np.uint32, 640 * 9),
    (np.uint16, None, 768 * 16),
]


@pytest.mark.parametrize("dtype,value,tile", TILES)
@pytest.mark.parametrize("d", [-1, 0, 1])
def test_sizes_around_one_tile_per_cta(oracle, dtype, value, tile, d):
    rng = np.random.default_rng(11 + d)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    # the tile of the build at hand may be smaller or larger: sizes on both sides of each multiple
    for n in sorted({sms * tile + d, sms * tile // 2 + d, sms * tile * 2 + d, 3 * tile + d, 5121 + d}):
        k = I.uniform_bits(np.dtype(f"u{np.dtype(dtype).itemsize}"), n, rng).view(dtype)
        if np.dtype(dtype).kind == "f":
            k = rng.standard_normal(n).astype(dtype)
        v = None if value is None else I.index_values(n, value)
        ko, vo, _ = gpu_sort(k, v)[:3]
        rk, rv = oracle.radix_sort(k, v, threads=8)
        assert ko.tobytes() == rk.tobytes()
        assert v is None or vo.tobytes() == rv.tobytes()


@pytest.mark.parametrize("n", [3001, 50021, 1 << 20])
@pytest.mark.parametrize("captured", [False, True])
def test_between_writer_and_reader(oracle, n, captured):
    """A kernel writes the keys, the sort follows, a kernel reads its output, eight times over the
    same buffers on one stream, without a wait on the host."""
    from cccl_gb300 import SortOrder, make_radix_sort

    rng = np.random.default_rng(n)
    base = I.uniform_bits(np.uint32, n, rng)
    src = to_dev(base)
    ki, ko = torch.empty_like(src), torch.empty_like(src)
    vi = torch.arange(n, dtype=torch.int32, device="cuda")
    vo = torch.empty_like(vi)
    args = dict(d_in_keys=ki, d_out_keys=ko, d_in_values=vi, d_out_values=vo)
    s = make_radix_sort(order=SortOrder.ASCENDING, **args)
    temp = torch.empty(s(temp_storage=None, num_items=n, **args), dtype=torch.uint8, device="cuda")
    outs = torch.empty((8, 2, n), dtype=torch.int32, device="cuda")
    words = src.view(torch.int32)

    def steps():
        for i in range(8):
            torch.bitwise_xor(words, i * 0x01010101, out=ki.view(torch.int32))
            s(temp_storage=temp, num_items=n, **args)
            outs[i, 0].copy_(ko.view(torch.int32))
            outs[i, 1].copy_(vo)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        steps()
    side.synchronize()
    if captured:
        outs.zero_()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            steps()
        graph.replay()
    torch.cuda.synchronize()
    for i in range(8):
        rk, rv = oracle.radix_sort(base ^ np.uint32(i * 0x01010101), np.arange(n, dtype=np.int32), threads=8)
        assert from_dev(outs[i, 0], np.uint32).tobytes() == rk.tobytes()
        assert from_dev(outs[i, 1], np.int32).tobytes() == rv.tobytes()
