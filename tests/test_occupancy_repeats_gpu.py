"""Exact occupancy of values that come several times in a row (low-complexity sequence): runs within a warp's 32 values and
across its edges, equal values of different bins and different values of one bin beside them, against the sequential C
oracle; and a call of one value takes no longer than one of different values."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [1, 2, 5])
def test_occupancy_of_runs(gpu_lib, oracle, h):
    bins, rows = 70, 3001
    rng = np.random.default_rng(h)
    lens = np.concatenate([np.arange(1, 70), [31, 32, 33, 64, 1, 1, 300, 5000]])
    v = np.repeat(rng.integers(0, 200, lens.size, dtype=np.uint64), lens)
    b = np.repeat(rng.integers(0, bins, lens.size).astype(np.uint64), lens)
    b[2000:2040] = np.arange(40) % bins  # one value, another bin each
    v[2100:2140] = np.arange(40)         # one bin, another value each
    g = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(rows), hg.hash_function_count(h), True)
    o = oracle.ibf(bins, rows, h, True)
    for n in (1, 31, 32, 33, 1000, v.size, v.size):
        g.emplace_many(v[:n], b[:n])
        o.emplace(v[:n], b[:n])
        np.testing.assert_array_equal(g.occupancy, o.occupancy())
        np.testing.assert_array_equal(g.words(), o.words())


def test_one_value_takes_no_longer_than_many(gpu_lib):
    import time

    import torch

    n = 1 << 20
    took = {}
    for name, v in (("many", torch.arange(n, dtype=torch.int64) * 0x9E3779B97F4A7C1), ("one", torch.full((n,), 5))):
        d = v.cuda()
        g = hg.interleaved_bloom_filter(hg.bin_count(64), hg.bin_size(1 << 22), hg.hash_function_count(2), True)
        times = []
        for _ in range(6):
            g.clear(np.arange(64, dtype=np.uint64))
            torch.cuda.synchronize()
            t = time.perf_counter()
            N.call("hibf_gpu_ibf_emplace_d", g._h, d.data_ptr(), None, n, 3, None)  # returns when it is done
            times.append(time.perf_counter() - t)
        took[name] = min(times)
    assert took["one"] < 2 * took["many"] + 3e-4, took
