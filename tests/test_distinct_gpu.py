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


def _took(inputs):
    """Seconds of build_inputs, the fastest of three, and its last results."""
    import time

    cfg = B.config(input_fn=lambda u, it: it.push(inputs[u]), number_of_user_bins=len(inputs))
    layout, times = _layout(len(inputs)), []
    for _ in range(3):
        t = time.perf_counter()
        got = B.build_inputs(cfg, layout)
        times.append(time.perf_counter() - t)
    return min(times), got


@pytest.mark.parametrize("values", ["dense", "ranges", "one"])
def test_dense_and_repeated_values_take_no_longer(gpu_lib, values):
    """User bins of the same small values, of neighbouring ranges of ids and of one value each against random ones: 2^24
    values in 4,096 bins.  Hashed alike, the ranges took a second and more on the device."""
    rng = np.random.default_rng(3)
    bins, n = 4096, 4096
    random = [rng.integers(0, 1 << 64, n, dtype=np.uint64) for _ in range(bins)]
    make = {"dense": lambda u: rng.permutation(n).astype(np.uint64) << np.uint64(14),
            "ranges": lambda u: rng.permutation(n).astype(np.uint64) + np.uint64(u << 17),
            "one": lambda u: np.full(n, u >> 6, np.uint64)}[values]
    inputs = [make(u) for u in range(bins)]
    base, _ = _took(random)
    took, (offs, vals) = _took(inputs)
    assert took < 2 * base + 0.1, (took, base)
    if values == "one":
        np.testing.assert_array_equal(offs, np.arange(bins + 1))
        np.testing.assert_array_equal(vals, np.arange(bins) >> 6)
    else:
        np.testing.assert_array_equal(offs, np.arange(bins + 1) * n)
        np.testing.assert_array_equal(vals, np.concatenate(inputs))
