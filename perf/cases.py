"""The sorts this package is used for, as measurable cases.

A case names an operation and its input; every run is one call of a built sort with its
temporary storage already allocated, as a program that sorts repeatedly keeps them:

  radix      make_radix_sort(...)(...)      keys alone, or keys with values
  segmented  make_segmented_sort(...)(...)  many segments of one array, each sorted
  learned    make_learned_sort(...)(...)    the learned-partition form of a radix sort

Fields: ``key`` and ``value`` (types; value "" = keys alone), ``n`` (items), ``order``
("asc" or "desc"), ``dist`` (the keys' distribution, see ``_keys``), ``begin_bit`` and
``end_bit`` of a radix sort (end 0 = the whole key), ``mean`` and ``sigma`` of the lognormal
segment lengths (mean of ln(length)). Values are the items' original indices, which is what
an argsort carries.
"""

import math

import torch

import cccl_gb300 as G

_TYPES = {
    "f16": torch.float16,
    "i32": torch.int32,
    "u32": torch.uint32,
    "f32": torch.float32,
    "i64": torch.int64,
    "u64": torch.uint64,
    "f64": torch.float64,
}
_BYTES = {"": 0, "f16": 2, "i32": 4, "u32": 4, "f32": 4, "i64": 8, "u64": 8, "f64": 8}
_SIGNED = {2: torch.int16, 4: torch.int32, 8: torch.int64}


def _case(op, key, value, n, dist, order="asc", **more):
    case = {"op": op, "key": key, "value": value, "n": n, "dist": dist, "order": order}
    if op == "radix":
        case["begin_bit"] = 0
        case["end_bit"] = 0
    case.update(more)
    return case


def listed():
    cases = {
        # the smallest calls: one batch's scores argsorted, where launch latency is all
        "scores_f32_2k": _case("radix", "f32", "i32", 2000, "normal", order="desc"),
        # token, cell or particle ids of one step
        "ids_u32_50k": _case("radix", "u32", "", 50021, "uniform"),
        # half-precision scores with their positions
        "scores_f16_1m": _case("radix", "f16", "i32", 1000003, "normal", order="desc"),
        # 2^24 32-bit keys alone: the plain workload of the repository's benchmark
        "keys_u32_16m": _case("radix", "u32", "", 1 << 24, "uniform"),
        # the same at 2^28 keys
        "keys_u32_256m": _case("radix", "u32", "", 1 << 28, "uniform"),
        # float argsort of an odd size
        "argsort_f32_33m": _case("radix", "f32", "i32", 33333333, "normal"),
        # 2^28 64-bit keys with 32-bit indices: the benchmark's headline
        "pairs_u64_256m": _case("radix", "u64", "u32", 1 << 28, "uniform"),
        # the benchmark's low-entropy keys (AND of three uniform words), descending
        "pairs_u64_and3_64m": _case("radix", "u64", "u32", 1 << 26, "and3", order="desc"),
        # double-precision measurements with 64-bit row numbers
        "rows_f64_100m": _case("radix", "f64", "i64", 100000007, "normal"),
        # the benchmark's batched segmented sort: 2^27 pairs in segments of very uneven length
        "segments_f32_128m": _case("segmented", "f32", "i32", 1 << 27, "normal", mean=5.0, sigma=2.5),
        # adjacency lists or posting lists: many short rows of integer ids, keys alone
        "rows_i32_16m": _case("segmented", "i32", "", 16777213, "uniform", mean=5.0, sigma=0.8),
        # the learned-partition sort of skewed doubles with 64-bit values
        "learned_f64_256m": _case("learned", "f64", "i64", 1 << 28, "lognormal"),
    }
    return [dict(case, name=name) for name, case in cases.items()]


# what the listed cases move at most: 2^28 items of 16 bytes, read once and written once
_MOST_BYTES = 2 * 16 * (1 << 28)


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["radix", "radix", "radix", "radix", "segmented", "learned"])
    order = rng.choice(["asc", "asc", "desc"])
    if op == "learned":
        return _case(op, "f64", "i64", _log_uniform(rng, 1 << 21, 1 << 28), rng.choice(["lognormal", "mix"]), order)
    if op == "segmented":
        key, value = rng.choice([("f32", "i32"), ("i32", ""), ("f32", ""), ("i64", "i32")])
        dist = "normal" if key == "f32" else "uniform"
        mean = rng.uniform(3.0, 6.0)
        return _case(op, key, value, _log_uniform(rng, 1 << 16, 1 << 27), dist, order, mean=mean,
                     sigma=rng.uniform(0.5, 2.5))
    key = rng.choice(["f16", "u32", "i32", "f32", "i64", "u64", "f64"])
    value = rng.choice(["", "i32", "i32", "i64"])
    most = min(1 << 28, _MOST_BYTES // (2 * (_BYTES[key] + _BYTES[value])))
    n = _log_uniform(rng, 1000, most)
    if key in ("f16", "f32", "f64"):
        return _case(op, key, value, n, rng.choice(["normal", "normal", "lognormal"]), order)
    case = _case(op, key, value, n, rng.choice(["uniform", "uniform", "and3", "below"]), order)
    if rng.random() < 0.2:  # a partial bit window
        bits = 8 * _BYTES[key]
        case["begin_bit"] = rng.randrange(0, bits // 2)
        case["end_bit"] = rng.randrange(bits // 2 + 1, bits + 1)
    return case


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _random_bits(n, nbytes, g):
    words = (n * nbytes + 7) // 8
    w = torch.randint(-(1 << 63), (1 << 63) - 1, (words,), dtype=torch.int64, device="cuda", generator=g)
    return w.view(_SIGNED[nbytes])[:n]


def _keys(case, g):
    """The case's keys. Integers: ``uniform`` over the whole type; ``and3``, the bitwise AND of
    three uniform words (low entropy); ``below``, whole numbers below 2^20 (4-byte keys) or
    2^40 (8-byte keys), as ids and time stamps are. Floats: ``normal`` N(0, 1), 0.1 % of the
    keys +0.0 or -0.0; ``lognormal`` with sigma 2 (4-byte and smaller keys) or 3; ``mix``,
    half lognormal, half U(0, 1)."""
    n, key, dist = case["n"], case["key"], case["dist"]
    dtype, nbytes = _TYPES[key], _BYTES[key]
    if key[0] in "iu":
        k = _random_bits(n, nbytes, g)
        if dist == "and3":
            k = k & _random_bits(n, nbytes, g)
            k = k & _random_bits(n, nbytes, g)
        elif dist == "below":
            k = k & ((1 << (5 * nbytes)) - 1)
        return k.contiguous().view(dtype)
    make = torch.float64 if key == "f64" else torch.float32
    k = torch.randn(n, dtype=make, device="cuda", generator=g)
    if dist == "normal":
        zeros = max(1, n // 1000)
        at = torch.randint(0, n, (zeros,), device="cuda", generator=g)
        k[at] = 0.0
        k[at[: zeros // 2]] = -0.0
    else:
        k = torch.exp(k * (3.0 if key == "f64" else 2.0))
        if dist == "mix":
            uniform = torch.rand(n, dtype=make, device="cuda", generator=g)
            k = torch.where(torch.rand(n, device="cuda", generator=g) < 0.5, k, uniform)
    if key == "f16":
        k = k.clamp(-60000.0, 60000.0)
    return k.to(dtype)


def _offsets(case, seed):
    """Segment bounds of the whole array: lognormal lengths, every twentieth segment empty,
    drawn until the array is full (lengths of at most 2^23)."""
    n = case["n"]
    g = torch.Generator()
    g.manual_seed(seed + 1)
    at, parts, total = [0], [], 0
    mean_len = math.exp(case["mean"] + case["sigma"] ** 2 / 2)
    while total < n:
        count = max(1024, int(1.2 * (n - total) / mean_len))
        length = torch.exp(case["mean"] + case["sigma"] * torch.randn(count, generator=g, dtype=torch.float64))
        length = length.round().clamp(1, 1 << 23).to(torch.int64)
        length[torch.rand(count, generator=g) < 0.05] = 0
        parts.append(length)
        total += int(length.sum())
    ends = torch.cumsum(torch.cat(parts), 0)
    keep = int(torch.searchsorted(ends, torch.tensor(n)))
    ends = torch.cat([ends[:keep], torch.tensor([n])])
    return torch.cat([torch.tensor(at), ends]).to(torch.int32).cuda()


def prepare(case, seed):
    g = _generator(seed)
    keys = _keys(case, g)
    n = case["n"]
    values = values_out = None
    if case["value"]:
        signed = _SIGNED[_BYTES[case["value"]]]
        values = torch.arange(n, dtype=signed, device="cuda").view(_TYPES[case["value"]])
        values_out = torch.empty_like(values)
    arrays = dict(d_in_keys=keys, d_out_keys=torch.empty_like(keys), d_in_values=values, d_out_values=values_out)
    order = G.SortOrder.ASCENDING if case["order"] == "asc" else G.SortOrder.DESCENDING
    args = dict(arrays, num_items=n)
    if case["op"] == "segmented":
        offsets = _offsets(case, seed)
        bounds = dict(start_offsets_in=offsets[:-1], end_offsets_in=offsets[1:])
        sorter = G.make_segmented_sort(**arrays, **bounds, order=order)
        args.update(bounds, num_segments=offsets.numel() - 1)
    elif case["op"] == "learned":
        sorter = G.make_learned_sort(**arrays, order=order)
    else:
        sorter = G.make_radix_sort(**arrays, order=order)
        if case["end_bit"]:
            args.update(begin_bit=case["begin_bit"], end_bit=case["end_bit"])
    temp = torch.empty(max(1, sorter(temp_storage=None, **args)), dtype=torch.uint8, device="cuda")
    # unsigned arrays are handed back as their signed views, which more torch operations take
    outputs = tuple(
        t.view(_SIGNED[t.element_size()]) if not t.dtype.is_signed else t
        for t in (arrays["d_out_keys"], values_out)
        if t is not None
    )
    return {"sorter": sorter, "temp": temp, "args": args, "outputs": outputs if values is not None else outputs[0]}


def run(state):
    state["sorter"](temp_storage=state["temp"], **state["args"])
    return state["outputs"]


def work(case):
    """Every key and value read once and written once, every segment's two bounds read."""
    item = _BYTES[case["key"]] + _BYTES[case["value"]]
    moved = 2 * item * case["n"]
    if case["op"] == "segmented":
        moved += int(8 * case["n"] / math.exp(case["mean"] + case["sigma"] ** 2 / 2))
    return {"bytes": moved, "flops": 0}


def exact(case, seed):
    """Sorted floating-point keys by torch's sort in double precision; integer keys and the
    values are whole numbers."""
    if case["key"][0] in "iu":
        return None
    keys = _keys(case, _generator(seed)).to(torch.float64)
    descending = case["order"] == "desc"
    if case["op"] == "segmented":
        offsets = _offsets(case, seed).to(torch.int64)
        segment = torch.repeat_interleave(torch.arange(offsets.numel() - 1, device="cuda"), offsets[1:] - offsets[:-1])
        keys, by = torch.sort(keys, descending=descending)
        segment, by = torch.sort(segment[by], stable=True)
        keys = keys[by]
    else:
        keys = torch.sort(keys, descending=descending)[0]
    return (keys, None) if case["value"] else keys
