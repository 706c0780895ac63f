"""Rows wider than a warp (more than 2,048 technical bins), counted and ANDed in slabs of 32 words, and summation
segments of many bins: single-level counts and containment, and hierarchies with such an IBF, against the C oracle."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N
from hibf_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [2048, 2049, 2113, 2240, 3000, 4095, 6144 + 17 * 64])
@pytest.mark.parametrize("h", [1, 2, 5])
def test_wide_ibf_counts_and_contains(gpu_lib, oracle, bins, h):
    """Slab edges: a full slab, one word over, last slabs of 1, 2, 4, 15, 31 -> 32 and 17 -> 32 words; calls shorter
    than a warp's pass, at its edges, and long enough for flushes between (more than 124 values per lane)."""
    rows = 211
    g = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(rows), hg.hash_function_count(h))
    o = oracle.ibf(bins, rows, h)
    vals = S.stream_range(bins + h, 0, 40_000)
    to = (np.arange(vals.size, dtype=np.uint64) * np.uint64(7919)) % np.uint64(bins)
    g.emplace_many(vals, to)
    o.emplace(vals, to)
    for n in (1, 31, 32, 33, 127, 129, 65_003):
        q = np.concatenate([vals[: n // 2], S.stream_range(5, 0, n - n // 2)])
        np.testing.assert_array_equal(g.counting_agent(4).bulk_count(q), o.bulk_count(q, 4))
        np.testing.assert_array_equal(g.containment_agent().bulk_contains_words(q[:300]), o.bulk_contains(q[:300]))
    np.testing.assert_array_equal(g.counting_agent(1).bulk_count(q), o.bulk_count(q, 1))


@pytest.mark.parametrize("bins", [513, 577, 960, 1024, 1025, 2048, 2100])
@pytest.mark.parametrize("h", [1, 2])
def test_counts_by_asynchronous_copies(gpu_lib, oracle, bins, h):
    """Calls on both sides of the size from which rows of 9 words or more go through shared memory (200,000 pieces of 16
    words): 9, 10, 15, 16 words, last slabs of 1, 16 and 1 words; a tail of one value and of seven."""
    rows, slabs = 401, (bins + 1023) // 1024
    g = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(rows), hg.hash_function_count(h))
    o = oracle.ibf(bins, rows, h)
    vals = S.stream_range(bins + h, 0, 60_000)
    to = (np.arange(vals.size, dtype=np.uint64) * np.uint64(7919)) % np.uint64(bins)
    g.emplace_many(vals, to)
    o.emplace(vals, to)
    edge = -(-200_000 // slabs)
    q = np.concatenate([vals, S.stream_range(6, 0, 400_000)])
    for n in (edge - 1, edge, edge + 7, 300_001):
        np.testing.assert_array_equal(g.counting_agent(4).bulk_count(q[:n]), o.bulk_count(q[:n], 4, threads=8))


def _one_ibf(oracle, user_bin, rows, h, words):
    bins = user_bin.size
    n_ub = int(user_bin[user_bin < N.BIN_DELETED].max()) + 1
    t = dict(n_user_bins=n_ub, bins=np.array([bins], np.uint64), bin_size=np.array([rows], np.uint64),
             hash_funs=np.array([h], np.uint64), next_ibf=np.zeros(bins, np.uint64), user_bin=user_bin)
    H = hg.hierarchical_interleaved_bloom_filter.from_tables(n_ub, t["bins"], t["bin_size"], t["hash_funs"],
                                                             t["next_ibf"], t["user_bin"], words=[words])
    return H, oracle.hibf(dict(t, words=[words]))


@pytest.mark.parametrize("block", [0, 1 << 30])
@pytest.mark.parametrize("bins,split", [(2049, 1), (2112, 33), (3000, 40), (6400, 64)])
def test_hierarchy_with_a_wide_ibf(gpu_lib, oracle, bins, split, block):
    """Segments of one bin, of 33 and 40 bins (starting and ending inside a warp's 32 bins) and of 64, with deleted
    bins among them; membership (early exit) and wrapping 16-bit counts."""
    rng = np.random.default_rng(bins)
    group = np.arange(bins) // split
    group[rng.choice(bins - 1, 20, replace=False)] = -1
    # a deleted bin ends a run, and every run is a user bin of its own (a user bin has one place in a hierarchy)
    starts = (group >= 0) & (np.concatenate([[-1], group[:-1]]) != group)
    user_bin = np.where(group >= 0, np.cumsum(starts) - 1, 0).astype(np.uint64)
    user_bin[group < 0] = N.BIN_DELETED
    rows, words_per_row = 301, (bins + 63) // 64
    fill = rng.integers(0, 1 << 63, rows * words_per_row, dtype=np.uint64) & rng.integers(
        0, 1 << 63, rows * words_per_row, dtype=np.uint64)
    H, O = _one_ibf(oracle, user_bin, rows, 2, fill)
    lens = np.array([1, 40, 300, 777, 2000, 5000])
    qo = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    vals = rng.integers(0, 1 << 63, int(qo[-1]), dtype=np.uint64)
    # thresholds around the sums' expectation (an eighth of the bits pass both rows), so some pass and some do not
    for share in (0.03, 0.0625, 0.07):
        thr = np.maximum(1, np.floor(lens * share * split)).astype(np.uint64) % np.uint64(1 << 16)
        thr = np.maximum(thr, 1).astype(np.uint64)
        for schedule in (N.SCHEDULE_QUEUE, N.SCHEDULE_LEVELS):
            a = H.membership_agent()
            a.tuning = dict(a.tuning, block_queries=block, schedule=schedule, early_exit_min=1, early_exit_step=1)
            offs, ids, _ = a.query_batch(vals, qo, thr)
            o_off, o_ids = O.membership_batch(vals, qo, thr, threads=2)
            np.testing.assert_array_equal(offs, o_off)
            np.testing.assert_array_equal(ids, o_ids)
            c = H.counting_agent(2)
            c.tuning = dict(a.tuning)
            offs, ids, cnts = c.query_batch(vals, qo, thr)
            for i in range(lens.size):
                dense = np.zeros(H.number_of_user_bins, np.uint16)
                dense[ids[offs[i]:offs[i + 1]].astype(np.int64)] = cnts[offs[i]:offs[i + 1]]
                v = vals[int(qo[i]):int(qo[i + 1])]
                np.testing.assert_array_equal(dense, O.bulk_count(v, int(thr[i]), 2))


def test_sums_beyond_32_bits_use_the_wide_form(gpu_lib, oracle):
    """A user bin over 6,400 bins and a query of 400,000 values: its sum can pass 2^31, so the 64-bit scans answer.
    All-ones rows: the sum is 6,400 * 400,000 = 2.56e9."""
    bins, n = 6400, 400_000
    H, O = _one_ibf(oracle, np.zeros(bins, np.uint64), 64, 1, np.full(64 * 100, ~np.uint64(0), np.uint64))
    vals = S.stream_range(3, 0, n)
    qo = np.array([0, n], np.uint64)
    c = H.counting_agent(8)
    for thr in (bins * n, bins * n + 1):
        for block in (0, 1 << 30):
            c.tuning = dict(c.tuning, block_queries=block)
            offs, ids, cnts = c.query_batch(vals, qo, np.array([thr], np.uint64))
            assert list(cnts) == ([bins * n] if thr == bins * n else [])
            assert list(ids) == [0] * len(cnts)
    a = H.membership_agent()
    a.tuning = dict(a.tuning, block_queries=0)
    thr = np.array([bins * n % (1 << 16)], np.uint64)  # the 16-bit sum wraps to exactly this
    assert list(a.query_batch(vals, qo, thr)[1]) == [0]
    assert list(a.query_batch(vals, qo, thr + np.uint64(1))[1]) == []
