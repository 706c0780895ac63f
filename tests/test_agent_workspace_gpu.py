"""An agent's workspace when it cannot grow: a reserve that no device can hold is reported as OUT_OF_MEMORY, and the
batches after it -- small and general host batches, device batches -- answer as before it.  And when it grows: a captured
batch and the last batch's results, which lie in the buffers before, are gone and say so; its work counters and times
stay, as they do when a batch is captured, which runs nothing."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N
from tests import golden_io as G

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    d = G.hibf_case("synth600")
    t = G.tables(d)
    H = hg.hierarchical_interleaved_bloom_filter.from_tables(t["n_user_bins"], t["bins"], t["bin_size"], t["hash_funs"],
                                                             t["next_ibf"], t["user_bin"], words=t["words"])
    return d, H


def _batch(d, nq):
    """nq of the stored queries, over and over."""
    qv, qo = d["q_values"], d["q_offsets"].astype(np.int64)
    pick = np.arange(nq) % (qo.size - 1)
    vals = np.concatenate([qv[qo[i]:qo[i + 1]] for i in pick])
    return (vals, np.concatenate([[0], np.cumsum(qo[pick + 1] - qo[pick])]).astype(np.uint64),
            np.asarray(d["mem_t"])[pick].astype(np.uint64))


def _device(a, b):
    import torch

    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in b]
    torch.cuda.synchronize()
    a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), b[1].size - 1, dev[2].data_ptr())
    return a.fetch_results(b[1].size - 1)


def _same(got, want):
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])


@pytest.mark.parametrize("schedule", [N.SCHEDULE_QUEUE, N.SCHEDULE_LEVELS])
@pytest.mark.parametrize("queries,tasks,results", [(1 << 45, 1, 1), (1, 1 << 45, 1), (1, 1, 1 << 45), (1 << 63, 1, 1),
                                                   (1, 1 << 61, 1), (1, 1, 1 << 62)])
def test_batches_after_a_failed_reserve(gpu_lib, case, schedule, queries, tasks, results):
    """2^45 entries are 140 TB and more; 2^61 and above times an entry's bytes pass 2^64."""
    d, H = case
    small, large = _batch(d, 40), _batch(d, 3000)
    want_small, want_large = H.membership_agent().query_batch(*small), H.membership_agent().query_batch(*large)
    for first in ("small", "large", "device"):
        a = H.membership_agent()
        a.tuning = dict(a.tuning, schedule=schedule)
        _same(a.query_batch(*large), want_large)
        _same(a.query_batch(*small), want_small)  # leaves the workspace as the next small batch wants it
        with pytest.raises((N.HibfGpuError, MemoryError)) as e:
            a.reserve(queries, 16, tasks, results)
        assert not isinstance(e.value, hg.InvalidArgument)
        steps = {"small": lambda: _same(a.query_batch(*small), want_small),
                 "large": lambda: _same(a.query_batch(*large), want_large),
                 "device": lambda: _same(_device(a, large), want_large)}
        steps[first]()
        for step in steps.values():
            step()


@pytest.mark.parametrize("grow", ["queries", "tasks", "results", "host batch", "small batch", "device batch"])
def test_a_captured_batch_ends_with_its_workspace(gpu_lib, case, grow):
    import torch

    d, H = case
    b = _batch(d, 2000)
    want = H.membership_agent().query_batch(*b)
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in b]
    torch.cuda.synchronize()
    nq = b[1].size - 1
    a = H.membership_agent()
    a.reserve(nq, 16, 20_000, int(want[0][-1]) + 1)
    for _ in range(2):
        with pytest.raises(hg.InvalidArgument):
            a.fetch_results(nq)  # no batch has run
        a.capture_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), nq, dev[2].data_ptr())
        with pytest.raises(hg.InvalidArgument):
            a.fetch_results(nq)  # a capture runs nothing
        for _ in range(2):
            a.replay()
            _same(a.fetch_results(nq), want)
        if grow == "host batch":
            a.query_batch(*_batch(d, 9000))
        elif grow == "small batch":  # 100 queries that report every user bin outgrow the results
            s = _batch(d, 100)
            a.query_batch(s[0], s[1], np.zeros(100, np.uint64))
        elif grow == "device batch":  # its queries outgrow the agent's; the results it makes room for may not do
            big = [torch.from_numpy(x.view(np.int64)).cuda() for x in _batch(d, 9000)]
            torch.cuda.synchronize()
            a.query_batch_device(big[0].data_ptr(), big[1].data_ptr(), 9000, big[2].data_ptr())
            torch.cuda.synchronize()
        else:
            a.reserve(*[(1 << 17 if k == grow else 1) for k in ("queries", "values", "tasks", "results")])
        with pytest.raises(hg.InvalidArgument):
            a.replay()
        if grow in ("queries", "results"):
            with pytest.raises(hg.InvalidArgument):
                a.fetch_results(nq)
        elif grow == "tasks":  # the results stayed where they were
            _same(a.fetch_results(nq), want)
        a.capture_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), nq, dev[2].data_ptr())
        a.replay()
        _same(a.fetch_results(nq), want)
        a = H.membership_agent()
        a.reserve(nq, 16, 20_000, int(want[0][-1]) + 1)


@pytest.mark.parametrize("schedule", [N.SCHEDULE_QUEUE, N.SCHEDULE_LEVELS])
def test_last_work_outlives_growth_and_captures(gpu_lib, case, schedule):
    import torch

    d, H = case
    sizes = {"small": 40, "large": 3000}
    b = {k: _batch(d, n) for k, n in sizes.items()}
    dev = {k: [torch.from_numpy(x.view(np.int64)).cuda() for x in v] for k, v in b.items()}
    torch.cuda.synchronize()

    def agent():
        a = H.membership_agent()
        a.tuning = dict(a.tuning, schedule=schedule, block_queries=1024)
        a.reserve(3000, 16, 20_000, 200_000)
        return a

    def seen(a):
        return a.last_work(), a.last_work_executed(), a.level_work()

    def capture(a, k):
        a.capture_batch_device(dev[k][0].data_ptr(), dev[k][1].data_ptr(), sizes[k], dev[k][2].data_ptr())

    def timed(a):
        return a.kernel_ms(), a.level_ms(), a.last_timeline()

    fresh = agent()
    assert fresh.last_work() == (0, 0) and fresh.last_work_executed() == 0 and fresh.level_work() == []
    fresh.status()
    want = {}
    for k in sizes:
        a = agent()
        a.query_batch(*b[k])
        want[k] = seen(a)
        assert want[k][0][0] >= sizes[k]
    assert bool(want["large"][2]) == (schedule == N.SCHEDULE_LEVELS) and want["small"][2] == []
    for k in sizes:
        for other in sizes:
            a = agent()
            a.query_batch(*b[k])
            times = timed(a)
            a.reserve(5000, 16, 30_000, 300_000)  # before the counters were asked for
            assert seen(a) == want[k]
            capture(a, other)
            assert seen(a) == want[k] and timed(a) == times
            a.replay()
            assert seen(a) == want[other]
            a.query_batch(*b[k])
            assert seen(a) == want[k]
            a.replay()
            a.status()
            assert seen(a) == want[other]


def test_timeline_is_of_the_last_host_batch(gpu_lib, case):
    import torch

    d, H = case
    small, large = _batch(d, 40), _batch(d, 3000)
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in large]
    torch.cuda.synchronize()
    for many in (False, True):  # 40 queries that report all 600 user bins take the general result passes
        a = H.membership_agent()
        a.reserve(3000, 16, 20_000, 200_000)
        thr = np.zeros(40, np.uint64) if many else small[2]
        a.query_batch(*large)
        a.query_batch(small[0], small[1], thr)
        t = a.last_timeline()
        assert len(t) == 4 and t[0] == t[1] == 0.0 and 0.0 < t[2] <= t[3]
        a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), 3000, dev[2].data_ptr())
        a.status()
        assert a.last_timeline() == t
