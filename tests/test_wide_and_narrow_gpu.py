"""A hierarchy whose widest IBF needs more than 48 KiB of shared counters (3,000 bins: 94 KiB; 6,400 bins: 200 KiB, the most
there is) goes on answering after others with the same number of hash functions were made: the kernels are the same."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _flat(bins, h, seed):
    words = np.random.default_rng(seed).integers(0, 1 << 63, 301 * ((bins + 63) // 64), dtype=np.uint64)
    return hg.hierarchical_interleaved_bloom_filter.from_tables(
        bins, np.array([bins], np.uint64), np.array([301], np.uint64), np.array([h], np.uint64),
        np.zeros(bins, np.uint64), np.arange(bins, dtype=np.uint64), words=[words])


@pytest.mark.parametrize("h", [1, 3, 4])
@pytest.mark.parametrize("bins", [3000, 6400])
def test_wide_hierarchy_beside_a_narrow_one(gpu_lib, h, bins):
    import torch

    rng = np.random.default_rng(h)
    lens = np.array([1, 40, 300, 777])
    qo = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    vals = rng.integers(0, 1 << 63, int(qo[-1]), dtype=np.uint64)
    thr = np.maximum(1, (lens * 0.5 ** h).astype(np.uint64))
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in (vals, qo, thr)]
    torch.cuda.synchronize()
    wide = _flat(bins, h, 1)

    def answers():
        got = []
        for block, schedule in ((1 << 30, N.SCHEDULE_QUEUE), (0, N.SCHEDULE_QUEUE), (0, N.SCHEDULE_LEVELS)):
            a = wide.counting_agent(4)
            a.tuning = dict(a.tuning, block_queries=block, schedule=schedule)
            got.extend(a.query_batch(vals, qo, thr))
        got.append(wide.membership_agent().membership_for(vals[:300], int(thr[2])))
        features = torch.zeros((lens.size, 6), dtype=torch.float32, device="cuda")
        a.query_features(dev[0].data_ptr(), dev[1].data_ptr(), lens.size, dev[2].data_ptr(), 64, features.data_ptr())
        torch.cuda.synchronize()
        got.append(features.cpu().numpy())
        return got

    before = answers()
    narrow = _flat(64, h, 2)
    narrow.membership_agent().query_batch(vals, qo, thr)
    for x, y in zip(answers(), before):
        np.testing.assert_array_equal(x, y)
