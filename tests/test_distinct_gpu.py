"""Every user bin's distinct values in first-appearance order from the device's hash table, where it has edges: bins of
one value, of one value many times over, around a warp and a block, equal values in different bins, the values 0 and
2^64 - 1 (no value is reserved)."""

import numpy as np
import pytest

from hibf_gb300 import build as B

pytestmark = pytest.mark.gpu


def _layout(n):
    head = "#TOP_LEVEL_IBF fullest_technical_bin_idx:0\n#USER_BIN_IDX\tTECHNICAL_BIN_INDICES\tNUMBER_OF_TECHNICAL_BINS\n"
    return head + "".join(f"{u}\t{u}\t1\n" for u in range(n))


@pytest.mark.parametrize("seed", [1, 2])
def test_distinct_values_in_first_appearance_order(gpu_lib, seed):
    rng = np.random.default_rng(seed)
    top = np.uint64((1 << 64) - 1)
    inputs = [np.array([7], np.uint64), np.full(1000, top, np.uint64), np.zeros(33, np.uint64),
              np.array([top, 0, top, 1, 0], np.uint64)]
    for n in (31, 32, 33, 255, 257, 100_000):
        inputs.append(rng.integers(0, max(2, n // 2), n).astype(np.uint64))
    inputs.append(inputs[-1][::-1].copy())
    inputs.append(rng.integers(0, 1 << 64, 200_000, dtype=np.uint64))
    cfg = B.config(input_fn=lambda u, it: it.push(inputs[u]), number_of_user_bins=len(inputs))
    offs, vals = B.build_inputs(cfg, _layout(len(inputs)))
    for u, v in enumerate(inputs):
        _, first = np.unique(v, return_index=True)
        np.testing.assert_array_equal(vals[int(offs[u]):int(offs[u + 1])], v[np.sort(first)], err_msg=f"user bin {u}")
