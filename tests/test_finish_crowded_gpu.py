"""Pieces of the partition and finish (cccl_gb300/csrc/finish_kernels.cuh) in which a few bins hold many keys:
copies of one key around the sizes at which the form changes, a few or many different keys in one
place, several crowded bins of one warp; against the oracle, byte for byte, and where it is
known, whether the large form had to take pieces."""

import numpy as np
import pytest

import inputs as I

pytestmark = pytest.mark.gpu

MIN8 = 1 << 22  # finish_min_items in sort_policy.h
MIN4 = 1 << 26


def _control(temp, key_bytes):
    """FinishControl::route and large_pieces, behind the control block (radix_plan.h)."""
    at = (16432 + 4 * key_bytes + 255) // 256 * 256
    words = temp[at : at + 48].cpu().numpy().view(np.uint32)
    return int(words[0]), int(words[6])


def _plant(keys, rng, groups):
    """Puts every group of keys at places of their own, in random order."""
    places = rng.permutation(keys.size)
    at = 0
    for g in groups:
        keys[places[at : at + g.size]] = g
        at += g.size
    return keys


def _groups(case, rng):
    base = I.uniform_bits(np.uint64, 40, rng)
    one = np.uint64(1)
    if case.startswith("copies"):
        return [np.full(int(case[6:]), b) for b in base]
    if case == "a_few_others":  # copies of a key and two or three that share its place
        return [np.concatenate([np.full(150, b), b ^ np.arange(1, 3 + i % 2, dtype=np.uint64)]) for i, b in enumerate(base)]
    if case == "many_others":  # different keys in one place
        return [b & ~np.uint64(0xFFFFF) | I.uniform_bits(np.uint64, 200, rng) & np.uint64(0xFFFFF) for b in base]
    if case == "side_by_side":  # bins of one warp: 2^-14 of the key range apart
        return [np.full(90, (b & ~np.uint64(0xFF << 56)) + (one * np.uint64(j) << np.uint64(36))) for b in base for j in range(5)]
    raise ValueError(case)


@pytest.mark.parametrize(
    "case,large",
    [("copies64", False), ("copies65", False), ("copies128", False), ("copies129", False), ("copies300", False),
     ("copies512", None), ("copies513", True), ("copies700", True), ("a_few_others", None), ("many_others", False),
     ("side_by_side", None)],
)
def test_eight_byte_keys(oracle, case, large):
    from cccl_gb300 import sort_status
    from cccl_gb300._bindings import CUDA_SUCCESS
    from gpu_util import gpu_sort

    for i, (n, dtype, values, descending) in enumerate(((MIN8 + 5, np.uint64, np.uint32, False), (MIN8 + 6, np.int64, None, True),
                                                        (MIN8 + 7, np.float64, np.uint64, False))):
        rng = np.random.default_rng(100 + i)
        keys = I.uniform_bits(np.uint64, n, rng)
        groups = _groups(case, rng)
        keys = _plant(keys, rng, groups).view(dtype)
        if dtype == np.float64:
            keys[np.isnan(keys)] = 0.5
        v = None if values is None else I.index_values(n, values)
        ko, vo, _, temp = gpu_sort(keys, v, descending=descending, return_temp=True)
        assert sort_status(temp) == (CUDA_SUCCESS, 0)
        rk, rv = oracle.radix_sort(keys, v, descending=descending, threads=8)
        assert ko.tobytes() == rk.tobytes()
        assert v is None or vo.tobytes() == rv.tobytes()
        route, pieces = _control(temp, 8)
        if dtype != np.float64:
            assert route == 1
            if large is not None:
                assert (pieces > 0) == large


@pytest.mark.parametrize("dtype,values", [(np.uint32, None), (np.int32, np.uint32), (np.float32, None), (np.float32, np.uint64)])
def test_four_byte_keys(oracle, dtype, values):
    """Copies, zeros of both signs among them, in keys of evenly spread bits."""
    from cccl_gb300 import sort_status
    from cccl_gb300._bindings import CUDA_SUCCESS
    from gpu_util import gpu_sort

    rng = np.random.default_rng(7)
    n = MIN4 + 4097
    keys = I.uniform_bits(np.uint32, n, rng)
    copies = [np.full(c, b, np.uint32) for c, b in zip((64, 65, 100, 256, 450) * 40, I.uniform_bits(np.uint32, 200, rng))]
    zeros = np.where(np.arange(400) % 3 == 0, 0x80000000, 0).astype(np.uint32)
    keys = _plant(keys, rng, copies + [zeros]).view(dtype)
    if np.dtype(dtype).kind == "f":
        keys[np.isnan(keys)] = 0.5
    v = None if values is None else I.index_values(n, values)
    for descending in (False, True):
        ko, vo, _, temp = gpu_sort(keys, v, descending=descending, return_temp=True)
        assert sort_status(temp) == (CUDA_SUCCESS, 0)
        rk, rv = oracle.radix_sort(keys, v, descending=descending, threads=8)
        assert ko.tobytes() == rk.tobytes()
        assert v is None or vo.tobytes() == rv.tobytes()
        assert _control(temp, 4)[0] == 1
