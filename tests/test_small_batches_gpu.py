"""Small host batches (one copy in, the query kernel, one finishing block) against the general passes: at the edges of
the query and result counts where the path changes, and in any order of small, large, device, replayed and failed
batches on one agent, whose workspace the small ones leave ready for the next."""

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


def _batch(d, nq, seed, zero=()):
    """nq queries sampled from the stored ones; queries in `zero` report every user bin (threshold 0)."""
    rng = np.random.default_rng(seed)
    qv, qo = d["q_values"], d["q_offsets"].astype(np.int64)
    pick = rng.integers(0, qo.size - 1, nq)
    vals = np.concatenate([qv[qo[i]:qo[i + 1]] for i in pick])
    off = np.concatenate([[0], np.cumsum(qo[pick + 1] - qo[pick])]).astype(np.uint64)
    thr = np.asarray(d["mem_t"])[pick].astype(np.uint64)
    thr[list(zero)] = 0
    return vals, off, thr


def _general(H, b, mode=N.QUERY_MEMBERSHIP, width=2):
    """The same batch through the warp-per-task kernel and the general passes."""
    a = H.membership_agent()
    a.tuning = dict(a.tuning, block_queries=0)
    r = a.query_batch(*b, mode=mode, width=width)
    return r, a.last_work()


def _same(x, y):
    for i, (p, q) in enumerate(zip(x, y)):
        assert (p is None) == (q is None)
        if p is not None:
            np.testing.assert_array_equal(p, q, err_msg=f"result {i}")


@pytest.mark.parametrize("nq,zero", [(1, ()), (1, (0,)), (3, (0, 1, 2)), (4, (0, 1, 2, 3)), (31, ()), (33, (5,)),
                                     (1023, (7, 900)), (1024, (0, 1023)), (1025, (0,))])
def test_small_batches_equal_general_ones(gpu_lib, case, nq, zero):
    """600 user bins: 3 threshold-0 queries give 1,800 results, 4 give 2,400 (more than the finishing block takes)."""
    d, H = case
    b = _batch(d, nq, nq, zero)
    want, work = _general(H, b)
    a = H.membership_agent()
    for _ in range(3):
        _same(a.query_batch(*b), want)
        assert a.last_work() == work
        a.status()
    offs, ids, _ = a.fetch_results(nq)
    _same((offs, ids), want[:2])
    for width in (1, 2, 4, 8):
        c = (b[0], b[1], np.maximum(b[2] // np.uint64(2), 1))
        want_c, _ = _general(H, c, N.QUERY_COUNT, width)
        _same(H.counting_agent(width).query_batch(*c), want_c)


def test_one_agent_any_order_of_batches(gpu_lib, case):
    import torch

    d, H = case
    small, many, large = _batch(d, 50, 1), _batch(d, 40, 2, range(20)), _batch(d, 3000, 3)
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in large]
    torch.cuda.synchronize()
    nq = large[1].size - 1
    want = {k: _general(H, b) for k, b in (("small", small), ("many", many), ("large", large))}
    a = H.membership_agent()
    a.reserve(nq, large[0].size, nq * 16, nq * 64)
    a.capture_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), nq, dev[2].data_ptr())

    def check(k, got):
        _same(got[:2], want[k][0][:2])
        assert a.last_work() == want[k][1]

    def device():
        a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), nq, dev[2].data_ptr())
        return a.fetch_results(nq)

    def replayed():
        a.replay()
        return a.fetch_results(nq)

    steps = {"s": lambda: check("small", a.query_batch(*small)), "m": lambda: check("many", a.query_batch(*many)),
             "l": lambda: check("large", a.query_batch(*large)), "d": lambda: check("large", device()),
             "r": lambda: check("large", replayed())}
    for step in "ssmsslsdsrsmmsrrsdmls":
        steps[step]()
    v, o = small[0][:int(small[1][1])], int(small[2][0])
    single = a.membership_for(v, o)
    with pytest.raises(hg.InvalidArgument):
        a.query_batch(small[0], small[1], small[2] + np.uint64(1 << 16))
    np.testing.assert_array_equal(a.membership_for(v, o), single)
    steps["s"]()


def test_small_batch_outgrows_its_capacity(gpu_lib, case):
    """A fresh agent holds 4,096 results; 12 threshold-0 queries have 7,200: the batch grows it and starts over."""
    d, H = case
    b = _batch(d, 12, 5, range(12))
    a = H.membership_agent()
    want, _ = _general(H, b)
    for _ in range(2):
        _same(a.query_batch(*b), want)
    s = _batch(d, 9, 6)
    _same(a.query_batch(*s), _general(H, s)[0])


@pytest.mark.parametrize("nq", [1, 5, 152, 300])
@pytest.mark.parametrize("where", ["pageable", "pinned", "copied"])
def test_long_queries_in_small_batches(gpu_lib, case, nq, where):
    """Queries of hundreds to thousands of values (16 warps per block while an SM has one block at most), their values
    read in place from ordinary or page-locked memory (the roots leave them on the device for the lower levels) or
    copied first."""
    import torch

    d, H = case
    rng = np.random.default_rng(nq)
    qv, qo = d["q_values"], d["q_offsets"].astype(np.int64)
    vals, off, thr = [], [0], []
    for _ in range(nq):
        i = rng.integers(0, qo.size - 1)
        v = np.resize(qv[qo[i]:qo[i + 1]], int(rng.integers(600, 3000)))
        vals.append(v)
        off.append(off[-1] + v.size)
        thr.append(int(0.7 * v.size))
    b = (np.concatenate(vals), np.array(off, np.uint64), np.array(thr, np.uint64))
    want, work = _general(H, b)
    a = H.membership_agent()
    if where == "pinned":
        keep = torch.from_numpy(b[0].view(np.int64)).pin_memory()
        b = (keep.numpy().view(np.uint64), b[1], b[2])
    if where == "copied":
        a.set_host_read(False)
    for _ in range(3):
        _same(a.query_batch(*b), want)
        assert a.last_work() == work
    assert a.last_in_place() or where != "pinned"


@pytest.mark.parametrize("nq,zero", [(255, (254,)), (256, (0, 255)), (257, (256,)), (512, (256, 511))])
def test_finishing_block_has_a_thread_per_query(gpu_lib, case, nq, zero):
    """256 threads up to 256 queries, else 1,024; more results than threads in either."""
    d, H = case
    b = _batch(d, nq, nq, zero)
    a = H.membership_agent()
    want = _general(H, b)[0]
    for _ in range(2):
        _same(a.query_batch(*b), want)


@pytest.mark.parametrize("nq", [1025, 4095, 4096, 4097, 8193, 16383, 16384, 16385, 32769, 65535, 65536, 65537])
def test_result_offsets_of_many_queries(gpu_lib, case, nq):
    """Offsets by the one-block scan (pieces of 4,096 counts, four to a turn) and, past 65,536 queries, the three-launch
    one: a threshold-0 query gives every user bin, one above any possible count none."""
    d, H = case
    thr = np.full(nq, 65535, np.uint64)
    for q in {0, 1, 4094, 4095, 4096, 4097, 8191, 8192, 12287, 12288, 16383, 16384, 16385, 32768, 65535, nq - 1}:
        if q < nq:
            thr[q] = 0
    vals = np.random.default_rng(nq).integers(0, 1 << 63, nq, dtype=np.uint64)
    want = np.concatenate([[0], np.cumsum(np.where(thr == 0, 600, 0))])
    off, ids, _ = H.membership_agent().query_batch(vals, np.arange(nq + 1, dtype=np.uint64), thr)
    np.testing.assert_array_equal(off, want)
    np.testing.assert_array_equal(ids.reshape(-1, 600), np.tile(np.arange(600), (int(want[-1]) // 600, 1)))


def test_a_failed_small_batch_runs_once(gpu_lib):
    """Two IBFs that are each other's child: the descent ends at the hierarchy's depth and reports the cycle.  The times are
    those of the small batch (its start and its inputs at 0), not of a second run through the general path."""
    user_bin = np.arange(128, dtype=np.uint64)
    user_bin[[0, 64]] = N.BIN_MERGED
    user_bin = np.where(user_bin == N.BIN_MERGED, user_bin, np.arange(128, dtype=np.uint64) - 1)
    user_bin[65:] -= np.uint64(1)
    next_ibf = np.concatenate([np.zeros(64, np.uint64), np.ones(64, np.uint64)])
    next_ibf[[0, 64]] = (1, 0)
    ones = np.full(101, ~np.uint64(0), np.uint64)
    H = hg.hierarchical_interleaved_bloom_filter.from_tables(126, np.array([64, 64], np.uint64),
                                                             np.array([101, 101], np.uint64),
                                                             np.array([2, 2], np.uint64), next_ibf, user_bin,
                                                             words=[ones, ones])
    a = H.membership_agent()
    b = (np.arange(30, dtype=np.uint64), np.array([0, 10, 30], np.uint64), np.array([1, 1], np.uint64))
    for _ in range(2):
        with pytest.raises(hg.HibfGpuError) as e:
            a.query_batch(*b)
        assert e.value.status == N.ERR_CYCLE
        t = a.last_timeline()
        assert t[0] == t[1] == 0.0 and 0.0 < t[2] <= t[3]
        with pytest.raises(hg.HibfGpuError):
            a.status()
        high = (b[0], b[1], np.array([11, 21], np.uint64))  # more than a query has values: nothing to descend to
        assert a.query_batch(*high)[1].size == 0
        a.status()


@pytest.mark.parametrize("nq", [60, 700, 1023, 1300, 3000])
@pytest.mark.parametrize("n", [1535, 1536, 1537])
def test_descents_kept_and_queued(gpu_lib, case, nq, n):
    """Blocks that keep a task's first child or queue it (1,536 values; a block per query, several queries per block, and
    in between), with short queries between the long ones, as host and device batches."""
    import torch

    d, H = case
    rng = np.random.default_rng(nq + n)
    qv, qo = d["q_values"], d["q_offsets"].astype(np.int64)
    vals = []
    for k in range(nq):
        i = rng.integers(0, qo.size - 1)
        v = qv[qo[i]:qo[i + 1]]
        vals.append(v if k % 3 else np.resize(v, n))
    off = np.concatenate([[0], np.cumsum([v.size for v in vals])]).astype(np.uint64)
    b = (np.concatenate(vals), off, np.array([max(1, int(0.6 * v.size)) for v in vals], np.uint64))
    want, work = _general(H, b)
    a = H.membership_agent()
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in b]
    torch.cuda.synchronize()
    a.reserve(nq, 16, nq * 16 + 4096, nq * 64 + 4096)
    for _ in range(2):
        _same(a.query_batch(*b), want)
        assert a.last_work() == work
        a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), nq, dev[2].data_ptr())
        _same(a.fetch_results(nq), want)
