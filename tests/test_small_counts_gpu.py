"""bulk_count where its shape changes: one block or several per slab (256 values), values read in place or copied
(8,192), counts and containment words in the small host buffers or beyond (64 KiB), calls in a row on one filter (each
leaves the shared totals at 0), and after the filter was widened; host and device calls against the C oracle."""

import numpy as np
import pytest

import hibf_gb300 as hg
from hibf_gb300 import _native as N
from hibf_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins,h", [(1, 1), (64, 2), (130, 3), (1000, 5), (2050, 2), (9000, 2)])
def test_counts_at_the_edges_of_their_shapes(gpu_lib, oracle, bins, h):
    import torch

    rows = 997
    g = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(rows), hg.hash_function_count(h))
    o = oracle.ibf(bins, rows, h)
    vals = S.stream_range(bins, 0, 9000)
    to = (np.arange(vals.size) % bins).astype(np.uint64)
    g.emplace_many(vals, to)
    o.emplace(vals, to)
    q = np.concatenate([vals[:5000], S.stream_range(77, 0, 9000)])
    for n in (1, 8, 32, 33, 255, 256, 257, 513, 8191, 8192, 8193, 14_000, 250, 0, 257):
        for width in (1, 2, 4, 8):
            want = o.bulk_count(q[:n], width)
            np.testing.assert_array_equal(g.counting_agent(width).bulk_count(q[:n]), want, err_msg=f"{n} {width}")
        d_q = torch.from_numpy(q[:max(n, 1)].view(np.int64).copy()).cuda()
        out = torch.full((bins,), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        N.call("hibf_gpu_ibf_bulk_count_d", g._h, d_q.data_ptr(), n, 8, out.data_ptr(), None)
        N.call("hibf_gpu_ibf_status", g._h)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint64), want)
        for t in (0, 1, n // 4 + 1):
            np.testing.assert_array_equal(g.membership_agent().membership_for(q[:n], t), o.membership_for(q[:n], t))
        m = min(n, 2000)
        np.testing.assert_array_equal(g.containment_agent().bulk_contains_words(q[:m]), o.bulk_contains(q[:m]))
    wider = bins + 200
    g.increase_bin_number_to(hg.bin_count(wider))
    o.increase_bin_number_to(wider)
    for n in (250, 3000, 250):
        np.testing.assert_array_equal(g.counting_agent(2).bulk_count(q[:n]), o.bulk_count(q[:n], 2))
