"""Device batches on a caller's stream: read by the caller's own work on that stream without a synchronisation, and captured
into a graph of the caller's, which is replayed between the agent's other batches without the agent knowing."""

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


def _batch(d, nq, first=0):
    import torch

    qv, qo = d["q_values"], d["q_offsets"].astype(np.int64)
    pick = (first + np.arange(nq)) % (qo.size - 1)
    b = (np.concatenate([qv[qo[i]:qo[i + 1]] for i in pick]),
         np.concatenate([[0], np.cumsum(qo[pick + 1] - qo[pick])]).astype(np.uint64),
         np.asarray(d["mem_t"])[pick].astype(np.uint64))
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in b]
    torch.cuda.synchronize()
    return b, dev


class _device_array:
    def __init__(self, pointer, n, typestr):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(pointer, False), version=3, strides=None)


@pytest.mark.parametrize("nq", [3, 500, 9000, 70_000])
def test_results_are_ready_for_the_callers_next_work(gpu_lib, case, nq):
    import torch

    d, H = case
    stream = torch.cuda.Stream()
    a = H.counting_agent(4)
    a.reserve(nq, 16, nq * 16 + 4096, nq * 64 + 4096)
    ref = H.counting_agent(4)
    ref.reserve(nq, 16, nq * 16 + 4096, nq * 64 + 4096)
    got, want = [], []
    for k in range(6):  # the next batch overwrites the results as soon as they are copied on the stream
        b, dev = _batch(d, nq, 17 * k)
        want.append((ref.query_batch(*b, N.QUERY_COUNT, 4), dev))
    a.set_stream(stream.cuda_stream)
    with torch.cuda.stream(stream):
        for w, dev in want:
            n = int(w[0][-1])
            offs, ids, counts = a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), nq, dev[2].data_ptr(),
                                                     N.QUERY_COUNT, 4)
            got.append([torch.as_tensor(_device_array(p, m, t), device="cuda").clone()
                        for p, m, t in ((offs, nq + 1, "<i8"), (ids, n, "<i8"), (counts, n, "<i4"))])
    torch.cuda.synchronize()
    a.set_stream(None)
    for g, (w, _) in zip(got, want):
        for x, y in zip(g, w):
            np.testing.assert_array_equal(x.cpu().numpy().view(y.dtype), y)


@pytest.mark.parametrize("nq", [40, 3000])
def test_a_callers_graph_between_small_batches(gpu_lib, case, nq):
    import torch

    d, H = case
    small, _ = _batch(d, 25, 5)
    large, dev = _batch(d, nq)
    ref = H.membership_agent()
    want_small, want_large = ref.query_batch(*small), ref.query_batch(*large)
    work_large = ref.last_work()
    a = H.membership_agent()
    a.reserve(9000, 1 << 20, 50_000, 400_000)

    def check_small():
        for x, y in zip(a.query_batch(*small)[:2], want_small[:2]):
            np.testing.assert_array_equal(x, y)
        a.status()

    check_small()  # leaves the workspace as the next small batch wants it
    a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), nq, dev[2].data_ptr())  # everything is loaded
    a.status()
    check_small()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        a.set_stream(torch.cuda.current_stream().cuda_stream)
        a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), nq, dev[2].data_ptr())
    a.set_stream(None)
    check_small()
    for step in "rsrrssrs":
        if step == "s":
            check_small()
            continue
        graph.replay()
        torch.cuda.synchronize()
        for x, y in zip(a.fetch_results(nq)[:2], want_large[:2]):
            np.testing.assert_array_equal(x, y)
        assert a.last_work() == work_large
