"""Host batches whose arrays do not start at a multiple of eight bytes (views into a buffer that was read from a file), in
ordinary and page-locked memory, at sizes where aligned ones are packed, read in place, and fetched by the first kernel:
they are copied, and answer like aligned ones.  The single-level filter's host calls copy theirs as well, and the server
copies the values of requests that lie like that in a registered range."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N
from hibf_gb300 import synthetic as S
from tests import golden_io as G

pytestmark = pytest.mark.gpu


def _shifted(x, shift, pinned=False):
    """x at `shift` bytes past a multiple of eight."""
    if pinned:
        import torch

        raw = torch.empty(x.nbytes + 16, dtype=torch.uint8, pin_memory=True).numpy()
    else:
        raw = np.empty(x.nbytes + 16, np.uint8)
    start = -raw.ctypes.data % 8 + shift
    y = raw[start:start + x.nbytes].view(x.dtype)
    y[:] = x
    assert y.ctypes.data % 8 == shift % 8
    return y


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("nq", [1, 40, 900, 9000])
def test_unaligned_host_batches(gpu_lib, nq, pinned):
    d = G.hibf_case("synth600")
    t = G.tables(d)
    H = hg.hierarchical_interleaved_bloom_filter.from_tables(t["n_user_bins"], t["bins"], t["bin_size"], t["hash_funs"],
                                                             t["next_ibf"], t["user_bin"], words=t["words"])
    qv, qo = d["q_values"], d["q_offsets"].astype(np.int64)
    pick = np.arange(nq) % (qo.size - 1)
    vals = np.concatenate([qv[qo[i]:qo[i + 1]] for i in pick])
    off = np.concatenate([[0], np.cumsum(qo[pick + 1] - qo[pick])]).astype(np.uint64)
    thr = np.asarray(d["mem_t"])[pick].astype(np.uint64)
    want = H.membership_agent().query_batch(vals, off, thr)
    a = H.membership_agent()
    for which in ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1)):
        for shift in (1, 4):
            b = [_shifted(x, shift if w else 0, pinned) for x, w in zip((vals, off, thr), which)]
            got = a.query_batch(*b)
            np.testing.assert_array_equal(got[0], want[0])
            np.testing.assert_array_equal(got[1], want[1])
            assert not (which[0] and a.last_in_place())
            got = a.query_batch(b[0], b[1], np.maximum(thr // np.uint64(2), 1), N.QUERY_COUNT, 4)
            again = a.query_batch(vals, off, np.maximum(thr // np.uint64(2), 1), N.QUERY_COUNT, 4)
            for x, y in zip(got, again):
                np.testing.assert_array_equal(x, y)
    first = _shifted(vals[:int(off[1])], 4, pinned)
    np.testing.assert_array_equal(a.membership_for(first, int(thr[0])), a.membership_for(vals[:int(off[1])], int(thr[0])))


@pytest.mark.parametrize("n", [5, 8000, 30_000])
def test_unaligned_ibf_calls(gpu_lib, n):
    g = hg.interleaved_bloom_filter(hg.bin_count(200), hg.bin_size(5000), hg.hash_function_count(2), True)
    f = hg.interleaved_bloom_filter(hg.bin_count(200), hg.bin_size(5000), hg.hash_function_count(2), True)
    v = S.stream_range(4, 0, n)
    b = (np.arange(n) % 200).astype(np.uint64)
    f.emplace_many(v, b)
    u = _shifted(v, 4)
    g.emplace_many(u, _shifted(b, 4))
    np.testing.assert_array_equal(g.words(), f.words())
    np.testing.assert_array_equal(g.occupancy, f.occupancy)
    np.testing.assert_array_equal(g.counting_agent(2).bulk_count(u), f.counting_agent(2).bulk_count(v))
    np.testing.assert_array_equal(g.membership_agent().membership_for(u, 3), f.membership_agent().membership_for(v, 3))
    np.testing.assert_array_equal(g.containment_agent().bulk_contains_words(u),
                                  f.containment_agent().bulk_contains_words(v))


def test_unaligned_served_requests(gpu_lib):
    import torch

    from hibf_gb300.serve import server

    d = G.hibf_case("synth600")
    t = G.tables(d)
    H = hg.hierarchical_interleaved_bloom_filter.from_tables(t["n_user_bins"], t["bins"], t["bin_size"], t["hash_funs"],
                                                             t["next_ibf"], t["user_bin"], words=t["words"])
    agent = H.membership_agent()
    qv, qo, thr = d["q_values"], d["q_offsets"].astype(np.int64), np.asarray(d["mem_t"]).astype(np.uint64)
    raw = torch.empty(qv.nbytes + 16, dtype=torch.uint8, pin_memory=True).numpy()
    for shift in (0, 4):
        start = -raw.ctypes.data % 8 + shift
        raw[start:start + qv.nbytes] = qv.view(np.uint8)
        base = raw.ctypes.data + start
        srv = server(H, slots=1, max_batch_queries=4096, max_batch_values=1 << 20, admission_bytes=1 << 30)
        srv.register_host(raw.ctypes.data, raw.nbytes, already_pinned=True)
        reqs = [(qo[k], (qo[k:k + 8] - qo[k]).astype(np.uint64), thr[k:k + 7].copy()) for k in range(0, qo.size - 8, 7)]
        ids = [srv.submit_borrowed(base + 8 * int(first), o, th) for first, o, th in reqs]
        for rid, (first, o, th) in zip(ids, reqs):
            st, offs, res, _ = srv.wait_result(rid, 7)
            want = agent.query_batch(qv[first:first + int(o[-1])], o, th)
            assert st == 0
            np.testing.assert_array_equal(offs, want[0])
            np.testing.assert_array_equal(res, want[1])
        assert bool(srv.batch_log()[:, 11].any()) == (shift == 0)  # the aligned ones ran zero copy
        srv.close()
