"""A batch in a claim order (longest query first) on an index several times the size of L2: its kernel takes no longer than
in query order.  Workers that go on with their tasks' first children mix the levels' accesses there: on the 8,192-user-bin
layout at 5% of its user bin sizes (0.6 GB) that made the ordered batch 1.3 times as long.  And the ordered batches answer as
the unordered ones do."""

import numpy as np
import pytest

from hibf_gb300 import _native as N

pytestmark = pytest.mark.gpu


def test_order_costs_nothing_on_an_index_beyond_l2(gpu_lib):
    import torch

    from hibf_gb300 import build as B
    from hibf_gb300 import synthetic as S
    from hibf_gb300.workloads import HIBF8192 as wl

    sizes = np.maximum(1, np.floor(np.diff(wl.user_bin_offsets().astype(np.float64)) * 0.05)).astype(np.uint64)
    offs = S.offsets_of(sizes)
    cfg = B.config(number_of_user_bins=wl.n_user_bins, number_of_hash_functions=wl.h, maximum_fpr=wl.fpr)
    hibf = B.build_synthetic(cfg, wl.layout_text(), wl.query.seed, offs)
    n = 20_000
    qo, thr = wl.query_offsets(0, n)
    dev = [torch.from_numpy(x.view(np.int64)).cuda() for x in (wl.queries_host(offs, 0, n, qo), qo, thr)]
    longest = torch.from_numpy(np.argsort(-np.diff(qo.astype(np.int64)), kind="stable").astype(np.int32)).cuda()
    torch.cuda.synchronize()
    a = hibf.membership_agent()
    a.reserve(n, 16, n * 16, n * 16)
    for mode, width in ((N.QUERY_MEMBERSHIP, 2), (N.QUERY_COUNT, 4)):
        took, got = {}, {}
        for name, order in (("query order", None), ("longest first", longest)):
            a.set_order(order.data_ptr() if order is not None else None, n)
            times = []
            for _ in range(9):
                a.query_batch_device(dev[0].data_ptr(), dev[1].data_ptr(), n, dev[2].data_ptr(), mode, width)
                got[name] = a.fetch_results(n, mode, width)
                times.append(a.kernel_ms())
            took[name] = float(np.median(times[2:]))
        assert took["longest first"] < 1.1 * took["query order"], (mode, took)
        for x, y in zip(*got.values()):
            np.testing.assert_array_equal(x, y)
