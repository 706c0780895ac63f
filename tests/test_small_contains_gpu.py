"""Containment words of few values on rows wider than 16 words, where a warp takes 8 values instead of 32: around a warp's
and a block's values and on both sides of the call size from which it takes 32 again (one wave of warps: 8 values x 9,728
warps over all slabs on 152 SMs), against the C oracle."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [1025, 2047, 2049, 3200])
@pytest.mark.parametrize("h", [1, 3, 5])
def test_containment_of_few_values(gpu_lib, oracle, bins, h):
    import torch

    rows = 307
    g = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(rows), hg.hash_function_count(h))
    o = oracle.ibf(bins, rows, h)
    vals = S.stream_range(bins + h, 0, 30_000)
    to = (np.arange(vals.size, dtype=np.uint64) * np.uint64(7919)) % np.uint64(bins)
    g.emplace_many(vals, to)
    o.emplace(vals, to)
    q = np.concatenate([vals[:20_000], S.stream_range(9, 0, 40_000)])
    want = o.bulk_contains(q)
    slabs = -(-bins // 1024)
    edge = torch.cuda.get_device_properties(0).multi_processor_count * 64 // slabs * 8
    assert edge + 8 < q.size
    for n in (1, 7, 8, 9, 63, 64, 65, 71, 513, 4097, edge - 1, edge, edge + 1, edge + 8):
        np.testing.assert_array_equal(g.containment_agent().bulk_contains_words(q[:n]), want[:n], err_msg=str(n))
