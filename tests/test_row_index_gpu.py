"""Row indices: filters of fewer than 2^32 rows hash to 32-bit indices, larger ones to 64-bit ones.  Filters on both
sides of the line are built and queried on the device and compared with a sparse model of the same inserts (a dict of
the rows that have bits), the rows computed here from the hash's definition with Python integers."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N
from hibf_gb300 import synthetic as S

SEEDS = (13572355802537770549, 13043817825332782213, 10650232656628343401, 16499269484942379435, 4893150838803335377)
M64 = (1 << 64) - 1


def row_of(v: int, seed: int, bin_size: int) -> int:
    h = (v * seed) & M64
    h ^= h >> (64 - bin_size.bit_length())
    return (((h * 11400714819323198485) & M64) * bin_size) >> 64


def row_of_32(v: int, seed: int, bin_size: int) -> int:
    """The 32-bit form, step by step (device.cuh, hash_row32)."""
    m = (v * seed) & M64
    hi, lo = m >> 32, m & 0xFFFFFFFF
    lo ^= hi >> (64 - bin_size.bit_length() - 32)
    h = ((hi << 32 | lo) * 11400714819323198485) & M64
    low = ((h & 0xFFFFFFFF) * bin_size) >> 32
    return ((h >> 32) * bin_size + low) >> 32


def test_the_32_bit_form_selects_the_same_row():
    rng = np.random.default_rng(1)
    sizes = [1, 2, 3, 63, 64, 1000, (1 << 31) - 1, 1 << 31, (1 << 31) + 1, (1 << 32) - 1]
    sizes += [int(x) for x in rng.integers(1, 1 << 32, 50)]
    values = [0, 1, M64] + [int(x) for x in rng.integers(0, 1 << 64, 200, dtype=np.uint64)]
    for size in sizes:
        for v in values:
            for seed in SEEDS:
                assert row_of(v, seed, size) == row_of_32(v, seed, size) < size


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [(1 << 32) - 1, (1 << 32) + 12345])
def test_filters_around_2_32_rows(gpu_lib, rows):
    h, bins = 3, 64
    vals = S.stream_range(11, 0, 600)
    to = (np.arange(vals.size) % bins).astype(np.uint64)
    bits: dict[int, int] = {}
    for v, b in zip(vals.tolist(), to.tolist()):
        for seed in SEEDS[:h]:
            r = row_of(v, seed, rows)
            bits[r] = bits.get(r, 0) | 1 << b
    q = np.concatenate([vals[:400], S.stream_range(12, 0, 300)])
    words = []
    for v in q.tolist():
        w = M64
        for seed in SEEDS[:h]:
            w &= bits.get(row_of(v, seed, rows), 0)
        words.append(w)
    words = np.array(words, np.uint64)
    counts = np.array([int((words >> np.uint64(b) & np.uint64(1)).sum()) for b in range(bins)], np.uint32)
    assert counts.sum() >= 400

    ibf = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(rows), hg.hash_function_count(h))
    ibf.emplace_many(vals, to)
    np.testing.assert_array_equal(ibf.containment_agent().bulk_contains_words(q)[:, 0], words)
    np.testing.assert_array_equal(ibf.counting_agent(4).bulk_count(q), counts)
    del ibf

    user_bin = np.arange(bins, dtype=np.uint64)
    H = hg.hierarchical_interleaved_bloom_filter.from_tables(bins, [bins], [rows], h, np.zeros(bins, np.uint64), user_bin)
    for b in range(bins):
        H.emplace(0, vals[to == b], b)
    agent = H.counting_agent(4)
    for block, schedule, lanes in ((0, N.SCHEDULE_QUEUE, 1), (0, N.SCHEDULE_LEVELS, 2), (1 << 30, N.SCHEDULE_QUEUE, 1)):
        agent.tuning = dict(agent.tuning, block_queries=block, schedule=schedule, values_per_lane=lanes)
        offs, ids, cnts = agent.query_batch(q, np.array([0, q.size], np.uint64), np.array([1], np.uint64))
        dense = np.zeros(bins, np.uint32)
        dense[ids.astype(np.int64)] = cnts
        np.testing.assert_array_equal(dense, counts)
