"""One build used by several host threads at once, each with its own stream and temporary storage:
short sorts whose launches differ in shared memory, and whole keys beside a bit window."""

import threading

import numpy as np
import pytest
import torch

import inputs as I
from gpu_util import from_dev, to_dev

pytestmark = pytest.mark.gpu


def test_sizes_and_windows_side_by_side(oracle):
    from cccl_gb300 import SortOrder, make_radix_sort

    rng = np.random.default_rng(17)
    built = None
    jobs = []
    for n, begin_bit, end_bit in ((5000, 0, 64), (100_000, 0, 64), (300_011, 0, 64), (300_012, 8, 16)):
        k, v = I.uniform_bits(np.uint64, n, rng), I.index_values(n)
        ki, vi = to_dev(k), to_dev(v)
        args = dict(d_in_keys=ki, d_out_keys=torch.zeros_like(ki), d_in_values=vi, d_out_values=torch.zeros_like(vi),
                    num_items=n, begin_bit=begin_bit, end_bit=end_bit)
        if built is None:
            built = make_radix_sort(order=SortOrder.ASCENDING, **{a: args[a] for a in args if a.startswith("d_")})
        temp = torch.empty(max(1, built(temp_storage=None, **args)), dtype=torch.uint8, device="cuda")
        jobs.append((k, v, args, temp, torch.cuda.Stream(), begin_bit, end_bit))
    torch.cuda.synchronize()
    errors = []

    def work(job):
        _, _, args, temp, stream, _, _ = job
        try:
            for _ in range(300):
                built(temp_storage=temp, stream=stream, **args)
        except Exception as e:  # reported by the test's own thread
            errors.append(f"{args['num_items']} items: {e}")

    threads = [threading.Thread(target=work, args=(job,)) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert errors == []
    for k, v, args, _, _, begin_bit, end_bit in jobs:
        rk, rv = oracle.radix_sort(k, v, begin_bit=begin_bit, end_bit=end_bit, threads=8)
        assert from_dev(args["d_out_keys"], np.uint64).tobytes() == rk.tobytes()
        assert from_dev(args["d_out_values"], np.uint32).tobytes() == rv.tobytes()
