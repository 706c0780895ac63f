"""Results of batches in which some queries report every user bin (threshold 0) and the others none: the order of the long
segments where the passes deal the queries to blocks and turns (912 blocks; 8, then up to 256 queries of a block a turn),
and their time when the long ones are neighbours."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N
from tests import golden_io as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hibf():
    t = G.tables(G.hibf_case("synth600"))
    return hg.hierarchical_interleaved_bloom_filter.from_tables(t["n_user_bins"], t["bins"], t["bin_size"],
                                                                t["hash_funs"], t["next_ibf"], t["user_bin"],
                                                                words=t["words"])


def _device(nq, long):
    """One value per query; the queries in `long` report all 600 user bins."""
    import torch

    thr = np.full(nq, 65535, np.uint64)
    thr[long] = 0
    vals = np.random.default_rng(nq).integers(0, 1 << 63, nq, dtype=np.uint64)
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in (vals, np.arange(nq + 1, dtype=np.uint64), thr)]
    torch.cuda.synchronize()
    return dev, thr


def _run(a, dev):
    a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), dev[0].numel(), dev[2].data_ptr())


@pytest.mark.parametrize("nq", [1, 2, 8, 911, 912, 913, 1824, 7295, 7296, 7297, 29_185, 233_471, 233_472, 233_473, 300_000])
def test_long_segments_are_sorted_wherever_they_lie(gpu_lib, hibf, nq):
    at = {0, 1, 7, 8, 910, 911, 912, 913, 1823, 7295, 7296, nq // 2, nq // 2 + 1, nq - 2, nq - 1} | set(range(300, 340))
    dev, thr = _device(nq, sorted(q for q in at if 0 <= q < nq))
    a = hibf.membership_agent()
    n = int((thr == 0).sum())
    a.reserve(nq, 16, 4 * nq + 4096, 600 * n + 4096)
    _run(a, dev)
    offs, ids, _ = a.fetch_results(nq)
    np.testing.assert_array_equal(offs, np.concatenate([[0], np.cumsum(np.where(thr == 0, 600, 0))]))
    np.testing.assert_array_equal(ids.reshape(-1, 600), np.tile(np.arange(600), (n, 1)))


def test_neighbouring_long_segments_cost_what_spread_ones_do(gpu_lib, hibf):
    """256 queries of 30,000: neighbours against one in every 117.  One block sorting all of them took about 30 times as
    long as the blocks together."""
    import torch

    nq, n = 30_000, 256
    stream = torch.cuda.Stream()
    took = {}
    for name, long in (("spread", np.arange(n) * 117), ("neighbours", np.arange(n) + 1000)):
        dev, _ = _device(nq, long)
        a = hibf.membership_agent()
        a.set_stream(stream.cuda_stream)
        a.reserve(nq, 16, 8 * nq, 600 * n + 4096)
        times = []
        for _ in range(7):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record(stream)
            _run(a, dev)
            e[1].record(stream)
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]) - a.kernel_ms())
        took[name] = min(times)
        a.status()
        a.set_stream(None)
    assert took["neighbours"] < 3 * took["spread"] + 0.1, took
