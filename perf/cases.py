"""Performance cases of the framework: what its users have it do, through its public entry points.

Three directions: queries of a hierarchical filter (HIBF), queries of a single-level filter (IBF), and the inserts that
build or renew a filter.  Sizes are those of the workloads in hibf_gb300/workloads.py and of the benchmark, from a
single read to a whole batch of a million queries; every case is a plain dict and `draw` gives more of the same
ranges.  All data is the seeded synthetic stream of include/hibf_gb300_synthetic.h.

The filters are those of the workloads themselves (a layout belongs to its user bin sizes), so a query case's seed
chooses the queries, and states that live at the same time share one filter, as agents of one program do.  All
outputs are whole numbers (user bin ids, counts, bit words), so there is nothing that could be off by a rounding.
"""

from __future__ import annotations

import math
import weakref
from functools import lru_cache

import numpy as np
import torch

import hibf_gb300 as hg
from hibf_gb300 import _native as N
from hibf_gb300 import build as B
from hibf_gb300 import synthetic as S
from hibf_gb300 import workloads as W

IBF_FPR = 0.05


def listed() -> list[dict]:
    return [
        # one read (250 k-mer hashes) against a 64-bin single-level filter that L2 holds: the smallest call there is
        dict(name="ibf_read", kind="ibf_host", bins=64, rows=1 << 20, h=2, n=250, op="membership", width=2),
        # the same read against the 8,192-user-bin index, as seqan::hibf's per-query agent is called
        dict(name="hibf_read", kind="hibf", index="hibf8192", nq=1, op="single", length=250, width=2, source="host",
             levels=False),
        # a hundred reads at once from ordinary host arrays: an interactive request or a server's batch
        dict(name="hibf_batch100", kind="hibf", index="hibf8192", nq=100, op="membership", width=2, source="host",
             levels=False),
        # the 64-user-bin workload in full: 10,000 queries from ordinary host arrays
        dict(name="hibf64_batch", kind="hibf", index="hibf64", nq=10000, op="membership", width=2, source="host",
             levels=False),
        # counting agent, 32-bit counters, values already on the device (abundance estimates need the counts)
        dict(name="hibf_count", kind="hibf", index="hibf8192", nq=20011, op="count", width=4, source="device",
             levels=False),
        # host batch in page-locked memory, read in place by the kernel: the benchmark's end-to-end call
        dict(name="hibf_pinned", kind="hibf", index="hibf8192", nq=60000, op="membership", width=2, source="pinned",
             levels=True),
        # the benchmark's headline step: a million queries resident on the device
        dict(name="hibf_step", kind="hibf", index="hibf8192", nq=1000000, op="membership", width=2, source="device",
             levels=True),
        # h = 3 and rows of 64 to 256 bins: the 65,536-user-bin layout at a hundredth of its user bin sizes
        dict(name="hibf65536_step", kind="hibf", index="hibf65536", nq=100003, op="membership", width=2,
             source="device", levels=True),
        # the benchmark's single-level step: counts and containment words of 2^24 values over 1,024 bins, 8 GiB
        dict(name="ibf1024_step", kind="ibf_device", bins=1024, rows=1 << 26, h=3, n=1 << 24, op="both", width=2),
        # a flat filter over the 8,192 user bins instead of a hierarchy (rows of 1 KiB), 200,003 values
        dict(name="ibf8192_flat", kind="ibf_device", bins=8192, rows=1 << 20, h=2, n=200003, op="both", width=4),
        # 64 of a filter's user bins renewed in place: cleared, inserted again, occupancies kept
        dict(name="ibf_renew", kind="renew", bins=1024, rows=1 << 16, h=2, renewed=64, track=True),
        # an index built from a layout and an input function, the 64-user-bin workload in full
        dict(name="hibf64_build", kind="build", scale=1.0),
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return max(int(lo), min(int(hi), int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng) -> dict:
    """One more case of the ranges of `listed`: the same kinds, sizes over the logarithm of their range."""
    kind = rng.choice(["hibf", "hibf", "hibf", "ibf_host", "ibf_device", "ibf_device", "renew", "build"])
    if kind == "hibf":
        index = rng.choice(["hibf64", "hibf8192", "hibf8192", "hibf65536"])
        op = rng.choice(["single", "membership", "membership", "count"])
        source = "host" if op == "single" else rng.choice(["host", "device", "device", "pinned"])
        most = {"host": 10000, "pinned": 60000, "device": 200000 if index == "hibf8192" else 100003}[source]
        if op == "single":
            return dict(kind=kind, index=index, nq=rng.randint(1, 8), op=op, length=_log_int(rng, 20, 2000), width=2,
                        source=source, levels=False)
        return dict(kind=kind, index=index, nq=_log_int(rng, 2, most), op=op,
                    width=rng.choice([2, 4, 8]) if op == "count" else 2, source=source,
                    levels=rng.random() < 0.5)
    if kind in ("ibf_host", "ibf_device"):
        bins = _log_int(rng, 1, 8192)
        row_bytes = 8 * ((bins + 63) // 64)
        rows = _log_int(rng, 1 << 12, min(1 << 26, (8 << 30) // row_bytes))
        most = min(1 << 24, (2 << 30) // row_bytes) if kind == "ibf_device" else 20000
        return dict(kind=kind, bins=bins, rows=rows, h=rng.randint(1, 5), n=_log_int(rng, 1, most),
                    op=rng.choice(["membership", "count", "contains"] if kind == "ibf_host" else
                                  ["count", "contains", "both"]), width=rng.choice([1, 2, 4, 8]))
    if kind == "renew":
        bins = _log_int(rng, 1, 1024)
        return dict(kind=kind, bins=bins, rows=_log_int(rng, 1 << 10, 1 << 16), h=rng.randint(1, 5),
                    renewed=rng.randint(1, min(bins, 64)), track=rng.random() < 0.7)
    return dict(kind="build", scale=math.exp(rng.uniform(math.log(0.05), 0.0)))


# -- filters: one per workload, shared by the states that live at the same time ---------------------------------------
_SCALE = {"hibf64": 1.0, "hibf8192": 1.0, "hibf65536": 0.01}
_alive: "weakref.WeakValueDictionary[tuple, _shared]" = weakref.WeakValueDictionary()


class _shared:
    """A filter and what belongs to it; goes away with the last state that holds it."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def _once(key: tuple, make):
    got = _alive.get(key)
    if got is None:
        got = make()
        _alive[key] = got
    return got


@lru_cache(maxsize=None)
def _sizes(index: str) -> np.ndarray:
    sizes = np.diff(W.WORKLOADS[index].user_bin_offsets())
    return np.maximum(1, np.floor(sizes.astype(np.float64) * _SCALE[index])).astype(np.uint64)


@lru_cache(maxsize=None)
def _split_table(index: str):
    return W.WORKLOADS[index].split_table(S.offsets_of(_sizes(index)))[0]


def _config(wl, **kw) -> B.config:
    return B.config(number_of_user_bins=wl.n_user_bins, number_of_hash_functions=wl.h, maximum_fpr=wl.fpr, **kw)


def _hibf(index: str) -> _shared:
    def make():
        wl, offs = W.WORKLOADS[index], S.offsets_of(_sizes(index))
        f = B.build_synthetic(_config(wl), wl.layout_text(), wl.query.seed, offs, _split_table(index))
        return _shared(hibf=f, offs=offs, d_offs=torch.from_numpy(offs.view(np.int64)).cuda())

    return _once(("hibf", index), make)


def _values_per_bin(rows: int, h: int) -> int:
    """User bin size at which a bin of `rows` bits has the false positive rate IBF_FPR."""
    return max(1, int(-math.log(1.0 - IBF_FPR ** (1.0 / h)) * rows / h))


def _ibf(bins: int, rows: int, h: int) -> _shared:
    def make():
        f = hg.interleaved_bloom_filter(hg.bin_count(bins), hg.bin_size(rows), hg.hash_function_count(h))
        vpb = _values_per_bin(rows, h)
        N.call("hibf_gpu_synth_ibf_emplace", f._h, 1, vpb, 0, bins, None)
        N.call("hibf_gpu_ibf_status", f._h)
        return _shared(ibf=f, vpb=vpb)

    return _once(("ibf", bins, rows, h), make)


# -- inputs ------------------------------------------------------------------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    return {"hibf": _prepare_hibf, "ibf_host": _prepare_ibf, "ibf_device": _prepare_ibf, "renew": _prepare_renew,
            "build": _prepare_build}[case["kind"]](case, seed)


def _stream_at(seed: int, pos: np.ndarray) -> np.ndarray:
    with np.errstate(over="ignore"):
        return S.mix64_np(np.uint64(seed) + (pos.astype(np.uint64) + np.uint64(1)) * np.uint64(S.GAMMA))


def _read(rng, seed: int, begin: int, end: int, n: int, noise: float) -> np.ndarray:
    """n values of a user bin that holds [begin, end) of the stream, a share of them replaced by random ones."""
    v = _stream_at(seed, rng.integers(begin, end, n))
    return np.where(rng.random(n) < noise, rng.integers(0, 1 << 63, n, dtype=np.uint64), v)


def _prepare_reads(case, seed):
    """Single queries, each a read of one user bin as the workloads mix them (2% noise)."""
    f, wl, n = _hibf(case["index"]), W.WORKLOADS[case["index"]], case["length"]
    rng = np.random.default_rng(seed)
    reads = []
    for b in rng.integers(0, wl.n_user_bins, case["nq"]):
        reads.append(_read(rng, wl.query.seed, int(f.offs[b]), int(f.offs[b + 1]), n, 0.02))
    return dict(case=case, filter=f, agent=f.hibf.membership_agent(), reads=reads,
                thr=S.query_threshold(wl.query, n), ids=np.zeros((case["nq"], 64), np.uint64))


def _prepare_hibf(case, seed):
    if case["op"] == "single":
        return _prepare_reads(case, seed)
    f, wl, nq = _hibf(case["index"]), W.WORKLOADS[case["index"]], case["nq"]
    first = seed << 22  # every seed has queries of its own
    qo, thr = wl.query_offsets(first, nq)
    d_qo = torch.from_numpy(qo.view(np.int64)).cuda()
    d_v = torch.empty(int(qo[-1]), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    wl.queries_device(f.d_offs.data_ptr(), first, nq, d_qo.data_ptr(), d_v.data_ptr())
    torch.cuda.synchronize()
    count = case["op"] == "count"
    agent = f.hibf.counting_agent(case["width"]) if count else f.hibf.membership_agent()
    if case["levels"]:
        agent.tuning = dict(agent.tuning, schedule=N.SCHEDULE_LEVELS, level_values_per_lane=2 if wl.h == 2 else 0)
    agent.reserve(nq, int(qo[-1]), nq * 8 + 65536, nq * 16 + 65536)
    st = dict(case=case, filter=f, agent=agent, nq=nq, ids=np.zeros(2 * nq + 256, np.uint64),
              counts=np.zeros(2 * nq + 256 if count else 0, {2: np.uint16, 4: np.uint32, 8: np.uint64}[case["width"]]),
              mode=N.QUERY_COUNT if count else N.QUERY_MEMBERSHIP)
    if case["source"] == "device":
        st.update(v=d_v, qo=d_qo, thr=torch.from_numpy(thr.view(np.int64)).cuda())
    elif case["source"] == "pinned":
        v = torch.empty(d_v.numel(), dtype=torch.int64, pin_memory=True)
        v.copy_(d_v)
        st.update(v=v.numpy().view(np.uint64), keep=v, qo=qo, thr=thr)
    else:
        st.update(v=d_v.cpu().numpy().view(np.uint64), qo=qo, thr=thr)
    return st


def _prepare_ibf(case, seed):
    f, n = _ibf(case["bins"], case["rows"], case["h"]), case["n"]
    st = dict(case=case, filter=f, ibf=f.ibf)
    if case["kind"] == "ibf_host":  # a read of one bin with a quarter of its values changed
        rng = np.random.default_rng(seed)
        b = int(rng.integers(0, case["bins"]))
        st.update(v=_read(rng, 1, b * f.vpb, (b + 1) * f.vpb, n, 0.25), ids=np.zeros(case["bins"], np.uint64),
                  counting=f.ibf.counting_agent(case["width"]), containment=f.ibf.containment_agent(),
                  membership=f.ibf.membership_agent())
        return st
    words = f.ibf.bin_words
    d_v = torch.empty(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    N.call("hibf_gpu_synth_ibf_queries_d", 1, case["bins"], f.vpb, seed << 26, n, d_v.data_ptr(), None)
    torch.cuda.synchronize()
    dt = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[case["width"]]
    st["v"] = d_v
    if case["op"] != "contains":
        st["counts"] = torch.empty(case["bins"], dtype=dt, device="cuda")
    if case["op"] != "count":
        st["words"] = torch.empty((n, words), dtype=torch.int64, device="cuda")
    return st


def _prepare_renew(case, seed):
    vpb = _values_per_bin(case["rows"], case["h"])
    f = hg.interleaved_bloom_filter(hg.bin_count(case["bins"]), hg.bin_size(case["rows"]),
                                    hg.hash_function_count(case["h"]), track_occupancy=case["track"])
    bins = np.random.default_rng(seed).permutation(case["bins"])[:case["renewed"]].astype(np.uint64)
    f.emplace_many(S.ibf_bin_values(seed, vpb, 0, 0, case["bins"] * vpb),
                   np.repeat(np.arange(case["bins"], dtype=np.uint64), vpb))
    values = np.concatenate([S.ibf_bin_values(seed + 1, vpb, int(b)) for b in bins])
    return dict(case=case, ibf=f, bins=bins, values=values, of=np.repeat(bins, vpb))


def _prepare_build(case, seed):
    wl = W.HIBF64
    sizes = np.maximum(1, np.floor(_sizes("hibf64").astype(np.float64) * case["scale"])).astype(np.uint64)
    offs = S.offsets_of(sizes)
    rng = np.random.default_rng(seed)
    inputs = []
    for u in range(wl.n_user_bins):  # a sequence repeats some of its k-mers: one in ten comes twice
        v = S.user_bin_values(seed, offs, u)
        inputs.append(np.concatenate([v, v[rng.integers(0, v.size, v.size // 10)]]))
    return dict(case=case, inputs=inputs, layout=wl.layout_text())


# -- one pass ----------------------------------------------------------------------------------------------------------
def _keep(buffer: np.ndarray, got: np.ndarray) -> np.ndarray:
    """Results into the program's own array, which has one size for all inputs (the rest of it is 0)."""
    buffer[:got.size] = got
    buffer[got.size:got.size + 64] = 0
    return buffer


def run(st: dict):
    case = st["case"]
    kind, op = case["kind"], case.get("op")
    if kind == "hibf":
        a = st["agent"]
        if op == "single":
            for keep, read in zip(st["ids"], st["reads"]):
                _keep(keep, a.membership_for(read, st["thr"]))
            return st["ids"]
        if case["source"] == "device":
            a.query_batch_device(st["v"].data_ptr(), st["qo"].data_ptr(), st["nq"], st["thr"].data_ptr(), st["mode"],
                                 case["width"])
            offs, ids, counts = a.fetch_results(st["nq"], st["mode"], case["width"])
        else:
            offs, ids, counts = a.query_batch(st["v"], st["qo"], st["thr"], st["mode"], case["width"])
        return [offs, _keep(st["ids"], ids), None if counts is None else _keep(st["counts"], counts)]
    if kind == "ibf_host":
        if op == "membership":
            return _keep(st["ids"], st["membership"].membership_for(st["v"], max(1, case["n"] // 2)))
        if op == "count":
            return st["counting"].bulk_count(st["v"])
        return st["containment"].bulk_contains_words(st["v"])
    if kind == "ibf_device":
        out = []
        if op != "contains":
            N.call("hibf_gpu_ibf_bulk_count_d", st["ibf"]._h, st["v"].data_ptr(), case["n"], case["width"],
                   st["counts"].data_ptr(), None)
            out.append(st["counts"])
        if op != "count":
            N.call("hibf_gpu_ibf_bulk_contains_d", st["ibf"]._h, st["v"].data_ptr(), case["n"],
                   st["words"].data_ptr(), None)
            out.append(st["words"])
        return out
    if kind == "renew":
        f = st["ibf"]
        f.clear(st["bins"])
        f.emplace_many(st["values"], st["of"])
        return [f.occupancy, f.words()]
    cfg = _config(W.HIBF64, input_fn=lambda u, it: it.push(st["inputs"][u]))
    f = hg.hierarchical_interleaved_bloom_filter(cfg, st["layout"])
    return [f.words(k) for k in range(f.n_ibfs)]


# -- what a pass cannot do without ----------------------------------------------------------------------------------
def _sectors(bins: int) -> int:
    """Bytes of the 32-byte memory sectors that one row of `bins` bins covers."""
    return 32 * ((8 * ((bins + 63) // 64) + 31) // 32)


def work(case: dict) -> dict:
    """Bytes: every input value once, the rows it selects (in the root for a hierarchy, whose lower levels depend on
    the queries), every output once.  No arithmetic counts: the path hashes, reads and adds bits."""
    if case["kind"] == "hibf":
        wl = W.WORKLOADS[case["index"]]
        values = case["nq"] * case.get("length", (wl.query.len_lo + wl.query.len_hi) / 2)
        root = {"hibf64": 64, "hibf8192": 64, "hibf65536": 256}[case["index"]]
        return dict(bytes=values * (8 + wl.h * _sectors(root)) + case["nq"] * 32, flops=0)
    if case["kind"] in ("ibf_host", "ibf_device"):
        per = 8 + case["h"] * _sectors(case["bins"])
        words = 8 * ((case["bins"] + 63) // 64)
        b = 0.0
        if case["op"] != "contains":
            b += case["n"] * per + case["bins"] * case["width"]
        if case["op"] in ("contains", "both"):
            b += case["n"] * (per + words)
        return dict(bytes=b, flops=0)
    if case["kind"] == "renew":
        n = case["renewed"] * _values_per_bin(case["rows"], case["h"])
        store = case["rows"] * 8 * ((case["bins"] + 63) // 64)
        return dict(bytes=16.0 * n + 64.0 * n * case["h"] + 3.0 * store, flops=0)
    n = 1.1 * float(_sizes("hibf64").sum()) * case["scale"]
    return dict(bytes=8 * n + 64.0 * 2 * n + 2.9e6 * case["scale"], flops=0)


def exact(case: dict, seed: int):
    """Every output is a whole number, bit for bit the same on any correct path: there is no value in 64 bits that a
    result could be nearer to."""
    return None
