"""Forms of the partition and finish (cccl_gb300/csrc/finish_kernels.cuh) that few inputs reach, with the route
they take asserted: the rest as the whole array, the order-free first pass over 8-byte keys alone,
two portions of it, and floating-point keys of 4 bytes."""

import numpy as np
import pytest

import inputs as I

pytestmark = pytest.mark.gpu


def _control(temp, key_bytes, portions=1):
    """FinishControl::route, rest_items and large_pieces, behind the control block (radix_plan.h)."""
    at = (16432 + 4 * key_bytes * portions + 255) // 256 * 256
    words = temp[at : at + 48].cpu().numpy().view(np.uint32)
    return int(words[0]), int(words[10]), int(words[6])


def _sample_places(n):
    """finish_sample_place in sort_policy.h, for every key of the sample (finish_sample_items)."""
    samples = 8192 if n >= 1 << 24 else 4096 if n >= 1 << 23 else 2048
    half = 1
    while half < 16 and (1 << (2 * half)) < n:
        half += 1
    mask = np.uint32((1 << half) - 1)
    h = np.uint32(half)
    place = np.arange(samples, dtype=np.uint32)
    todo = np.ones(samples, bool)
    with np.errstate(over="ignore"):
        while todo.any():
            left, right = place >> h, place & mask
            for step in range(1, 5):
                f = (right + np.uint32(step * 0x9E3779B1 & 0xFFFFFFFF)) * np.uint32(0x2C1B3C6D)
                f = (f ^ (f >> np.uint32(12))) * np.uint32(0x297A2D39)
                f ^= f >> np.uint32(15)
                left, right = right, left ^ (f & mask)
            place = np.where(todo, left << h | right, place)
            todo = place >= n
    assert np.unique(place).size == samples
    return place


@pytest.mark.parametrize("low_byte", [0xFF, 0x00])  # eight or seven digits that vary
@pytest.mark.parametrize("values,descending,overwrite", [(np.uint32, False, False), (None, True, False), (np.uint64, False, True)])
def test_rest_is_the_whole_array(oracle, low_byte, values, descending, overwrite):
    """Evenly spread keys where the sample looks, one bucket of different keys everywhere else."""
    from cccl_gb300 import sort_status
    from cccl_gb300._bindings import CUDA_SUCCESS
    from gpu_util import gpu_sort

    n = (1 << 22) + 4099
    rng = np.random.default_rng(low_byte)
    keys = I.uniform_bits(np.uint64, n, rng)
    crowd = np.ones(n, bool)
    crowd[_sample_places(n)] = False
    keys[crowd] = keys[crowd] >> np.uint64(16) | np.uint64(0x5A5A) << np.uint64(48)
    keys &= ~np.uint64(0xFF) | np.uint64(low_byte)
    v = None if values is None else I.index_values(n, values)
    ko, vo, _, temp = gpu_sort(keys, v, descending=descending, overwrite=overwrite, return_temp=True)
    assert sort_status(temp) == (CUDA_SUCCESS, 0)
    route, rest, _ = _control(temp, 8)
    assert route == 1 and 2 * rest > n
    rk, rv = oracle.radix_sort(keys, v, descending=descending, threads=8)
    assert ko.tobytes() == rk.tobytes()
    assert v is None or vo.tobytes() == rv.tobytes()


@pytest.mark.parametrize("dtype,descending,overwrite", [(np.uint64, False, False), (np.int64, True, True)])
def test_order_free_first_pass_of_eight_byte_keys(oracle, dtype, descending, overwrite):
    from cccl_gb300 import sort_status
    from cccl_gb300._bindings import CUDA_SUCCESS
    from gpu_util import gpu_sort

    n = (1 << 26) + 7
    keys = I.uniform_bits(np.uint64, n, np.random.default_rng(3)).view(dtype)
    ko, _, _, temp = gpu_sort(keys, None, descending=descending, overwrite=overwrite, return_temp=True)
    assert sort_status(temp) == (CUDA_SUCCESS, 0)
    assert _control(temp, 8)[0] == 1
    rk, _ = oracle.radix_sort(keys, None, descending=descending, threads=8)
    assert ko.tobytes() == rk.tobytes()


def test_order_free_first_pass_in_two_portions():
    import torch

    from cccl_gb300 import SortOrder, make_radix_sort, sort_status
    from cccl_gb300._bindings import CUDA_SUCCESS

    n = (1 << 30) + 777
    torch.cuda.empty_cache()
    k = torch.empty(n, dtype=torch.int64, device="cuda")
    k.random_(-(1 << 63), (1 << 63) - 1, generator=torch.Generator(device="cuda").manual_seed(6))
    ko = torch.empty_like(k)
    args = dict(d_in_keys=k, d_out_keys=ko, d_in_values=None, d_out_values=None)
    s = make_radix_sort(order=SortOrder.ASCENDING, **args)
    temp = torch.empty(s(temp_storage=None, num_items=n, **args), dtype=torch.uint8, device="cuda")
    s(temp_storage=temp, num_items=n, **args)
    torch.cuda.synchronize()
    assert sort_status(temp) == (CUDA_SUCCESS, 0)
    assert _control(temp, 8, portions=2)[0] == 1
    del temp
    expected = torch.sort(k)[0]
    assert torch.equal(ko, expected)


@pytest.mark.parametrize("values", [None, np.uint32, np.uint64])
@pytest.mark.parametrize("descending,overwrite", [(False, True), (True, False)])
def test_four_byte_floats(oracle, values, descending, overwrite):
    """Evenly spread bits as floats, infinities and a few thousand zeros of both signs among them."""
    from cccl_gb300 import sort_status
    from cccl_gb300._bindings import CUDA_SUCCESS
    from gpu_util import gpu_sort

    n = (1 << 26) + 4099
    rng = np.random.default_rng(13)
    keys = I.uniform_bits(np.uint32, n, rng)
    places = rng.permutation(n)[:4000]
    keys[places] = np.where(np.arange(4000) % 2 == 0, 0x80000000, 0).astype(np.uint32)
    keys[places[:64]] = np.where(np.arange(64) % 2 == 0, 0xFF800000, 0x7F800000).astype(np.uint32)
    keys = keys.view(np.float32)
    keys[np.isnan(keys)] = 0.5
    v = None if values is None else I.index_values(n, values)
    ko, vo, _, temp = gpu_sort(keys, v, descending=descending, overwrite=overwrite, return_temp=True)
    assert sort_status(temp) == (CUDA_SUCCESS, 0)
    assert _control(temp, 4)[0] == 1
    rk, rv = oracle.radix_sort(keys, v, descending=descending, threads=8)
    assert ko.tobytes() == rk.tobytes()
    assert v is None or vo.tobytes() == rv.tobytes()
