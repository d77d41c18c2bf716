"""Partition and finish (cccl_gb300/csrc/finish_kernels.cuh): whole 4- and 8-byte keys sorted by
their top digits and finished in shared memory, against the oracle, byte for byte. The inputs
reach every part of it: pieces at the array's ends and of one bucket, even and uneven densities,
repeated keys, pieces that take the large form or LSD passes in shared memory, buckets that are
left to the rest kernel, and inputs whose sample asks for every digit pass."""

import numpy as np
import pytest

import inputs as I

pytestmark = pytest.mark.gpu

MIN8 = 1 << 22  # finish_min_items in sort_policy.h
MIN4 = 1 << 26


def _route(temp, key_bytes):
    """FinishControl::route and rest_items, behind the control block (radix_plan.h)."""
    at = (16432 + 4 * key_bytes + 255) // 256 * 256
    words = temp[at : at + 48].cpu().numpy().view(np.uint32)
    return int(words[0]), int(words[10])


def _keys(case, n, rng):
    u = I.uniform_bits(np.uint64, n, rng)
    if case == "uniform":
        return u
    if case == "normal":  # uneven densities, both tails, and a bucket of zeros
        k = rng.standard_normal(n)
        k[::1000] = 0.0
        k[5::1000] = -0.0
        return k
    if case == "specials":
        return I.with_specials(rng.lognormal(0.0, 3.0, n), rng, 1 / 64)
    if case == "below_2_40":  # three constant digits above the partition
        return u >> np.uint64(24)
    if case == "repeated":  # up to about 20 copies of a key, in one bin
        return I.uniform_bits(np.uint64, n // 16, rng)[rng.integers(0, n // 16, n)]
    if case == "hot":  # bins too full for the finish in many pieces
        k = u
        hot = rng.random(n) < 0.05
        k[hot] = u[rng.integers(0, 500, n)[hot]]
        return k
    if case == "one_in_fifty_equal":  # one bucket for the rest kernel, of one key
        k = u
        k[rng.random(n) < 0.02] = np.uint64(0x123456789ABCDEF0)
        return k
    if case == "clump":  # one bucket for the rest kernel, of different keys
        k = u
        m = rng.random(n) < 0.02
        k[m] = (np.uint64(0x1234) << np.uint64(48)) | (k[m] >> np.uint64(40))
        return k
    if case == "and3":  # every digit pass
        return u & I.uniform_bits(np.uint64, n, rng) & I.uniform_bits(np.uint64, n, rng)
    if case == "sorted":
        return np.sort(u)
    raise ValueError(case)


def _check(oracle, keys, values, descending, overwrite, route=None, rest=None):
    from cccl_gb300 import sort_status
    from cccl_gb300._bindings import CUDA_SUCCESS
    from gpu_util import gpu_sort

    ko, vo, sel, temp = gpu_sort(keys, values, descending=descending, overwrite=overwrite, return_temp=True)
    assert sort_status(temp) == (CUDA_SUCCESS, 0)
    if route is not None:
        got, left = _route(temp, keys.dtype.itemsize)
        assert got == route
        if rest is not None:
            assert (left > 0) == rest
    rk, rv = oracle.radix_sort(keys, values, descending=descending, threads=8)
    assert ko.tobytes() == rk.tobytes()
    if values is not None:
        assert vo.tobytes() == rv.tobytes()
    if overwrite:
        assert sel == 0


@pytest.mark.parametrize(
    "case,route,rest",
    [("uniform", 1, False), ("normal", 1, None), ("specials", None, None), ("below_2_40", 1, False),
     ("repeated", None, None), ("hot", None, None), ("one_in_fifty_equal", 1, True), ("clump", 1, True), ("and3", 0, None),
     ("sorted", 1, False)],
)
def test_eight_byte_keys(oracle, case, route, rest):
    rng = np.random.default_rng(len(case))
    for n, values, descending, overwrite in (
        (MIN8, np.uint32, False, False),
        (MIN8 + 1, None, True, False),
        (MIN8 + 12347, np.uint64, False, True),
    ):
        keys = _keys(case, n, rng)
        # an odd number of partition passes needs one more in a DoubleBuffer: the route may change
        _check(oracle, keys, None if values is None else I.index_values(n, values), descending, overwrite,
               None if overwrite else route, None if overwrite else rest)


@pytest.mark.parametrize("dtype,values", [(np.int64, np.uint32), (np.float64, np.uint64), (np.float64, None)])
def test_orders_and_kinds(oracle, dtype, values):
    rng = np.random.default_rng(7)
    n = 5_000_011
    keys = rng.standard_normal(n) if dtype == np.float64 else I.uniform_bits(np.uint64, n, rng).view(np.int64)
    for descending in (False, True):
        for overwrite in (False, True):
            _check(oracle, keys, None if values is None else I.index_values(n, values), descending, overwrite)


@pytest.mark.parametrize("dtype,values,descending", [(np.uint32, None, False), (np.int32, np.uint32, True),
                                                     (np.float32, None, True), (np.float32, np.uint64, False)])
def test_four_byte_keys(oracle, dtype, values, descending):
    rng = np.random.default_rng(11)
    n = MIN4 + 4099
    keys = I.uniform_bits(np.uint32, n, rng)
    route = 1
    if dtype == np.float32:  # U(0, 1) crowds into few top digits
        keys = np.where(keys < np.uint32(1 << 20), np.float32(0.0) * (keys % 2).astype(np.float32) * np.float32(-1.0),
                        keys.astype(np.float32))
        route = None
    _check(oracle, keys.view(dtype), None if values is None else I.index_values(n, values), descending, False, route)


def test_replayed_from_a_graph(oracle):
    """One captured sort, replayed on inputs of both routes."""
    import torch

    from cccl_gb300 import SortOrder, make_radix_sort
    from gpu_util import from_dev, to_dev

    rng = np.random.default_rng(3)
    n = MIN8 + 33
    k = to_dev(_keys("uniform", n, rng))
    v = to_dev(I.index_values(n))
    ko, vo = torch.empty_like(k), torch.empty_like(v)
    args = dict(d_in_keys=k, d_out_keys=ko, d_in_values=v, d_out_values=vo)
    sorter = make_radix_sort(order=SortOrder.ASCENDING, **args)
    temp = torch.empty(sorter(temp_storage=None, num_items=n, **args), dtype=torch.uint8, device="cuda")
    sorter(temp_storage=temp, num_items=n, **args)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sorter(temp_storage=temp, num_items=n, **args)
    for case, route in (("uniform", 1), ("and3", 0), ("clump", 1)):
        keys = _keys(case, n, rng)
        k.view(torch.uint8).copy_(torch.from_numpy(keys.view(np.uint8)))
        graph.replay()
        torch.cuda.synchronize()
        assert _route(temp, 8)[0] == route
        rk, rv = oracle.radix_sort(keys, I.index_values(n), threads=8)
        assert from_dev(ko, np.uint64).tobytes() == rk.tobytes() and from_dev(vo, np.uint32).tobytes() == rv.tobytes()


def test_two_portions():
    """More than 2^30 keys: the partition's passes run as two portions, and places in the pieces go
    beyond 2^30. A bucket of different keys at the array's end goes to the rest."""
    import torch
    from cccl_gb300 import SortOrder, make_radix_sort, sort_status
    from gpu_util import check_sorted_pairs

    n = (1 << 30) + 12345
    torch.cuda.empty_cache()
    gen = torch.Generator(device="cuda").manual_seed(5)
    k = torch.empty(n, dtype=torch.int64, device="cuda")
    k.random_(-(1 << 63), (1 << 63) - 1, generator=gen)
    k[12345 : n : 50] = k[12345 : n : 50] & 0xFFFFFFFFFF | (0x7FFF1234 << 32 & ~0xFFFFFFFFFF)
    v = torch.arange(n, dtype=torch.int32, device="cuda")
    ko, vo = torch.empty_like(k), torch.empty_like(v)
    args = dict(d_in_keys=k, d_out_keys=ko, d_in_values=v, d_out_values=vo)
    s = make_radix_sort(order=SortOrder.ASCENDING, **args)
    temp = torch.empty(s(temp_storage=None, num_items=n, **args), dtype=torch.uint8, device="cuda")
    s(temp_storage=temp, num_items=n, **args)
    torch.cuda.synchronize()
    sort_status(temp)
    route, rest = _route(temp, 8 * 2)
    assert route == 1 and rest > 0
    del temp
    assert check_sorted_pairs(k, ko, vo, "i")


@pytest.mark.parametrize("dist", ["uniform", "normal"])
def test_sorted_input_is_sampled_fairly(dist):
    """The sample sees the buckets of keys that are already in order as it does those of the same
    keys in any order, so the finish is left no large buckets."""
    import torch
    from cccl_gb300 import SortOrder, make_radix_sort
    from gpu_util import check_sorted_pairs

    n = (1 << 26) + 3
    gen = torch.Generator(device="cuda").manual_seed(9)
    k = torch.empty(n, dtype=torch.float64, device="cuda")
    k = k.normal_(generator=gen) if dist == "normal" else k.uniform_(generator=gen)
    light = []
    for keys in (k, torch.sort(k)[0]):
        v = torch.arange(n, dtype=torch.int32, device="cuda")
        ko, vo = torch.empty_like(keys), torch.empty_like(v)
        args = dict(d_in_keys=keys, d_out_keys=ko, d_in_values=v, d_out_values=vo)
        s = make_radix_sort(order=SortOrder.ASCENDING, **args)
        temp = torch.empty(s(temp_storage=None, num_items=n, **args), dtype=torch.uint8, device="cuda")
        s(temp_storage=temp, num_items=n, **args)
        torch.cuda.synchronize()
        at = (16432 + 4 * 8 + 255) // 256 * 256
        light.append(temp[at + 48 : at + 48 + 64].cpu().numpy().view(np.uint64).astype(np.int64))
        assert _route(temp, 8) == (1, 0)
        assert check_sorted_pairs(keys, ko, vo, "f")
    # pairs of three digits: some thousand, the same but for their spread
    assert abs(light[0][2] - light[1][2]) < 12 * np.sqrt(light[0][2]) + 12
