"""The scratch of inserts with exact occupancy, up to 122 MB a call, belongs to the device: many filters hold no more of
it than two, the last one gives it back, and filters of several threads insert at the same time."""

import gc
import threading

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import synthetic as S

pytestmark = pytest.mark.gpu

BINS, ROWS, H = 130, 50_000, 5


def _filter():
    return hg.interleaved_bloom_filter(hg.bin_count(BINS), hg.bin_size(ROWS), hg.hash_function_count(H), True)


def test_many_filters_share_their_scratch(gpu_lib):
    import torch

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free

    vals = S.stream_range(1, 0, 1 << 20)
    to = (np.arange(vals.size) % BINS).astype(np.uint64)
    _filter().emplace_many(vals[:100], to[:100])  # the kernels' own memory
    gc.collect()
    before = used()
    filters = [_filter() for _ in range(24)]
    for g in filters:
        g.emplace_many(vals, to)
    # per filter: 50,000 rows of 32 bytes and two input buffers of 8 MiB, each in pages of 2 MiB
    assert used() - before < 24 * (4 + 2 * 10 + 4) * (1 << 20) + 2 * 130 * (1 << 20)
    del filters, g
    gc.collect()
    assert used() - before < 32 << 20


def test_inserts_of_several_threads(gpu_lib, oracle):
    rng = np.random.default_rng(2)
    inputs = [(rng.integers(0, 60_000, n, dtype=np.uint64), rng.integers(0, BINS, n).astype(np.uint64))
              for n in (300_000, 1000, 120_000, 400_000)]
    want = []
    for v, b in inputs:
        o = oracle.ibf(BINS, ROWS, H, True)
        o.emplace(v, b)
        want.append(o.occupancy())
    got = [None] * len(inputs)

    def work(k):
        for _ in range(5):
            g = _filter()
            g.emplace_many(*inputs[k])
            got[k] = g.occupancy

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(inputs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for x, y in zip(got, want):
        np.testing.assert_array_equal(x, y)
