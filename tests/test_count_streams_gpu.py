"""hibf_gpu_ibf_bulk_count_d calls that overlap on one filter: on several streams, on more streams than the filter keeps
scratch for (16), from several threads on one stream, and a captured call replayed beside others.  Every call counts its own
values, so a total or a ticket of another call would show in its counts; they equal those of the same call alone."""

import threading

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N
from hibf_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def _filter(bins, h):
    g = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(1 << 14), hg.hash_function_count(h))
    vals = S.stream_range(bins, 0, 100_000)
    g.emplace_many(vals, (np.arange(vals.size) % bins).astype(np.uint64))
    return g, vals


def _calls(torch, g, vals, n_calls, n):
    """Inputs of n_calls different calls, their counts one after the other, and outputs to fill."""
    ins = [torch.from_numpy(np.roll(vals, 7919 * k)[: n - 37 * k].view(np.int64).copy()).cuda() for k in range(n_calls)]
    want = [torch.zeros(g.bin_count(), dtype=torch.int64, device="cuda") for _ in ins]
    torch.cuda.synchronize()
    for d, out in zip(ins, want):
        N.call("hibf_gpu_ibf_bulk_count_d", g._h, d.data_ptr(), d.numel(), 8, out.data_ptr(), None)
        N.call("hibf_gpu_ibf_status", g._h)
    return ins, want, [torch.full_like(w, -1) for w in want]


def _count(g, d, out, stream):
    N.call("hibf_gpu_ibf_bulk_count_d", g._h, d.data_ptr(), d.numel(), 8, out.data_ptr(), stream.cuda_stream)


@pytest.mark.parametrize("bins,h", [(64, 2), (1000, 3), (2050, 2)])
@pytest.mark.parametrize("n_streams", [2, 16, 19])
def test_counts_on_several_streams(gpu_lib, bins, h, n_streams):
    import torch

    g, vals = _filter(bins, h)
    ins, want, outs = _calls(torch, g, vals, n_streams, 60_000)
    streams = [torch.cuda.Stream() for _ in ins]
    for _ in range(30):
        for d, out, s in zip(ins, outs, streams):
            with torch.cuda.stream(s):
                out.fill_(-1)
            _count(g, d, out, s)
        torch.cuda.synchronize()
        for k, (out, w) in enumerate(zip(outs, want)):
            assert torch.equal(out, w), k


def test_counts_from_several_threads_on_one_stream(gpu_lib):
    import torch

    g, vals = _filter(1000, 3)
    ins, want, outs = _calls(torch, g, vals, 4, 60_000)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def work(k):
        for _ in range(50):
            _count(g, ins[k], outs[k], stream)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(ins))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for k, (out, w) in enumerate(zip(outs, want)):
        assert torch.equal(out, w), k


def test_captured_count_beside_others(gpu_lib):
    import torch

    g, vals = _filter(1000, 3)
    ins, want, outs = _calls(torch, g, vals, 2, 60_000)
    graph, replayed, direct = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        _count(g, ins[0], outs[0], torch.cuda.current_stream())
    for _ in range(30):
        with torch.cuda.stream(replayed):
            outs[0].fill_(-1)
            graph.replay()
        _count(g, ins[1], outs[1], direct)
        torch.cuda.synchronize()
        assert torch.equal(outs[0], want[0]) and torch.equal(outs[1], want[1])
