"""Occupancy of a filter that tracks it where the insert's chunks and its table of positions have edges: calls of one
value, around a warp, and around a chunk (2^20 values), with values repeated within and across calls and chunks and bins
that already hold bits, against the sequential C oracle."""

import numpy as np
import pytest

import hibf_gb300 as hg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [1, 2, 5])
@pytest.mark.parametrize("sizes,distinct", [((1, 31, 33, 257), 100), (((1 << 20) - 1, 2), 1 << 40),
                                            (((1 << 20) + 1, 1 << 20), 300_000)])
def test_occupancy_at_chunk_edges(gpu_lib, oracle, h, sizes, distinct):
    bins, rows = 130, 50_000
    rng = np.random.default_rng(h)
    g = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(rows), hg.hash_function_count(h), True)
    o = oracle.ibf(bins, rows, h, True)
    for n in sizes:
        v = rng.integers(0, distinct, n, dtype=np.uint64)
        b = rng.integers(0, bins, n).astype(np.uint64)
        g.emplace_many(v, b)
        o.emplace(v, b)
        np.testing.assert_array_equal(g.occupancy, o.occupancy())
    b[:] = 77  # one bin for all, once more: nothing new for values it has
    g.emplace_many(v, hg.bin_index(77))
    o.emplace(v, b)
    np.testing.assert_array_equal(g.occupancy, o.occupancy())
    np.testing.assert_array_equal(g.words(), o.words())
    with pytest.raises(hg.InvalidArgument):
        g.emplace_many(np.arange(5), np.array([0, 1, bins, 2, 3], np.uint64))
    many = np.zeros(40_000, np.uint64)  # checked on the device
    many[-1] = bins
    with pytest.raises(hg.InvalidArgument):
        g.emplace_many(np.arange(many.size), many)
    np.testing.assert_array_equal(g.words(), o.words())
    np.testing.assert_array_equal(g.occupancy, o.occupancy())
