"""Performance cases of the batch overlap queries, through the public entry points.

Every case is one call that a program makes against a built index: the device-buffer calls of the
C-ABI (queries and results resident in HBM), its host-buffer calls, or the numpy calls of
``GpuIndex``.  Result buffers are the caller's and a little larger than the result.
Sizes, contigs and length distributions are those of ``superintervals_gb300.workloads`` (its five
configurations), scaled where a full one would not fit the card three times over.

A case holds:
  op       what is called: search (contig-local positions, C++ order), values (payloads, descending),
           count, coverage, keys, intersect, difference, upper_bound -- device buffers;
           host_search -- the C-ABI search with pinned host buffers; lookup -- GpuIndex.search on
           numpy arrays; build -- a new index from numpy arrays and its arrays back
  bits     coordinate width, 32 or 64
  n, nq    intervals of the index, queries of the call
  contigs  "all" (24 human chromosomes), or names joined with "+"
  kind     interval lengths: "genes" (log-normal, median 500), "reads" (90% of 150 bp, 10% of
           10-50 kb), "deep" (log-normal, median 300, and 1% of 1-5 Mb), "hot" (starts 70% in
           Zipf hotspots, log-normal lengths, median 1000)
  ordered  queries sorted by start (else in random order)
"""
import ctypes as C
import math

import numpy as np
import torch

from superintervals_gb300.workloads import HUMAN_CONTIGS

LENGTHS = dict(HUMAN_CONTIGS)
# log-normal (median, sigma, longest) of the intervals and of the queries of each kind; and the
# share, shortest and longest of its long intervals
SHORT = {"genes": (500, 1.0, 100_000), "reads": None, "deep": (300, 1.5, 100_000), "hot": (1000, 1.0, 1_000_000)}
LONG = {"reads": (0.10, 10_000, 50_000), "deep": (0.01, 1_000_000, 5_000_000)}
READ = 150


def listed():
    return [
        # an interactive lookup: one region against a whole-genome annotation
        dict(name="lookup", op="lookup", bits=32, n=5_000_003, nq=1, contigs="all", kind="genes", ordered=False),
        # one request of a serving loop over a resident whole-genome index
        dict(name="serve", op="host_search", bits=32, n=20_000_011, nq=30_011, contigs="all", kind="genes",
             ordered=False),
        # a small annotation job, sparse hits: intervals and queries of one chromosome
        dict(name="small_search", op="search", bits=32, n=100_000, nq=100_000, contigs="chr1", kind="genes",
             ordered=False),
        # overlap counts of a whole-genome query set
        dict(name="count", op="count", bits=32, n=12_500_000, nq=12_500_000, contigs="all", kind="deep",
             ordered=False),
        # the headline search: about 500 hits a query, two chromosomes at the full density
        dict(name="search_dense", op="search", bits=32, n=7_950_001, nq=7_949_993, contigs="chr1+chr2", kind="deep",
             ordered=False),
        # payloads of reads against reads, queries in file (coordinate) order
        dict(name="values_reads", op="values", bits=32, n=10_000_000, nq=2_500_000, contigs="chr1", kind="reads",
             ordered=True),
        # keys of every hit with 64-bit coordinates
        dict(name="keys_64", op="keys", bits=64, n=4_000_037, nq=1_999_993, contigs="all", kind="genes",
             ordered=False),
        # positions only: 64-bit coordinates crowded into hotspots
        dict(name="upper_bound_64", op="upper_bound", bits=64, n=20_000_000, nq=20_000_000, contigs="span", kind="hot",
             ordered=False),
        # two interval sets intersected, subtracted, and the covered lengths of one under the other
        dict(name="intersect", op="intersect", bits=32, n=5_000_000, nq=5_000_000, contigs="all", kind="deep",
             ordered=False),
        dict(name="difference", op="difference", bits=32, n=5_000_000, nq=5_000_000, contigs="all", kind="genes",
             ordered=False),
        dict(name="coverage", op="coverage", bits=32, n=5_000_000, nq=5_000_000, contigs="all", kind="genes",
             ordered=False),
        # a new index from unsorted arrays, and its arrays back
        dict(name="build", op="build", bits=32, n=5_000_011, nq=0, contigs="all", kind="deep", ordered=False),
    ]


# most hits that a drawn case may have (the listed ones go to 4e9), by what one hit costs
MOST_HITS = {"search": 2e9, "values": 2e9, "keys": 3e8, "intersect": 3e8, "difference": 3e8, "host_search": 1e7, "lookup": 1e6}


def draw(rng):
    def size(a, b):
        return int(math.exp(rng.uniform(math.log(a), math.log(b))))

    op = rng.choice(["lookup", "host_search", "search", "search", "values", "count", "count", "keys", "intersect",
                     "difference", "coverage", "upper_bound", "build"])
    case = dict(op=op, bits=rng.choice([32, 32, 32, 64]), n=size(2_000, 12_500_000),
                nq={"lookup": size(1, 100), "host_search": size(100, 100_000), "build": 0}.get(op, size(500, 10_000_000)),
                contigs=rng.choice(["all", "all", "chr1", "chr21+chr22"]),
                kind=rng.choice(["genes", "reads", "deep"]), ordered=rng.random() < 0.25)
    if op in ("upper_bound", "count") and rng.random() < 0.4:
        case.update(bits=64, contigs="span", kind="hot")
    if op == "build":
        case["n"] = min(case["n"], 5_000_000)
    hits = expected_hits(case)
    if hits > MOST_HITS.get(op, 1e18):
        case["nq"] = max(1, int(case["nq"] * MOST_HITS[op] / hits))
    while op != "build" and expected_hits(case) < 8:  # something to find
        case["nq"] *= 2
    return case


# ---------------------------------------------------------------- inputs
def contig_lengths(case):
    if case["contigs"] == "span":
        return [3_100_000_000]
    if case["contigs"] == "all":
        return [ln for _, ln in HUMAN_CONTIGS]
    return [LENGTHS[c] for c in case["contigs"].split("+")]


def mean_lengths(case):
    """Mean length of an interval and of a query."""
    if SHORT[case["kind"]] is None:
        share, lo, hi = LONG["reads"]
        m = (1 - share) * READ + share * (lo + hi) / 2
        return m, m
    median, sigma, _ = SHORT[case["kind"]]
    short = median * math.exp(sigma * sigma / 2)
    if case["kind"] in LONG:
        share, lo, hi = LONG[case["kind"]]
        return (1 - share) * short + share * (lo + hi) / 2, short
    return short, short


def expected_hits(case):
    if case["kind"] == "hot":
        return 2.9e-3 * case["n"] * case["nq"]
    a, b = mean_lengths(case)
    return case["nq"] * (case["n"] / sum(contig_lengths(case))) * (a + b)


def per_contig(total, lens):
    """How many of `total` each contig gets, in proportion to its length."""
    cut = np.floor(np.cumsum(np.asarray(lens, np.float64)) / sum(lens) * total + 0.5).astype(np.int64)
    cut[-1] = total
    return np.diff(cut, prepend=0)


def lognormal(gen, n, kind):
    median, sigma, longest = SHORT[kind]
    z = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64)
    return torch.exp(math.log(median) + sigma * z).round_().clamp_(1, longest).to(torch.int64)


def uniform(gen, n, lo, hi):
    return (lo + torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * (hi - lo)).to(torch.int64)


def lengths(gen, n, kind, queries):
    if SHORT[kind] is None:
        ln = torch.full((n,), READ, dtype=torch.int64, device="cuda")
    else:
        ln = lognormal(gen, n, kind)
    if kind in LONG and not (queries and kind == "deep"):
        share, lo, hi = LONG[kind]
        is_long = torch.rand(n, generator=gen, device="cuda") < share
        ln = torch.where(is_long, uniform(gen, n, lo, hi + 1), ln)
    return ln


def starts(gen, case, n, contig):
    lens = torch.tensor(contig_lengths(case), dtype=torch.float64, device="cuda")
    u = torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)
    s = (u * lens[contig]).to(torch.int64)
    if case["kind"] == "hot":  # 70% in 10,000 hotspots of Zipf(1.1) weight, the same for intervals and queries
        spots = np.random.Generator(np.random.PCG64(3)).integers(0, int(lens[0]), 10_000)
        weight = np.cumsum(np.arange(1, 10_001, dtype=np.float64) ** -1.1)
        cdf = torch.from_numpy(weight / weight[-1]).cuda()
        pick = torch.searchsorted(cdf, torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)).clamp_(0, 9_999)
        jitter = torch.randn(n, generator=gen, device="cuda", dtype=torch.float64) * 5_000.0
        hot = torch.from_numpy(spots).cuda()[pick] + jitter.round_().to(torch.int64)
        s = torch.where(torch.rand(n, generator=gen, device="cuda") < 0.7, hot, s)
        s = s.clamp_(0, int(lens[0]) - 1)
    return s


def make_inputs(case, seed):
    """Intervals grouped by contig (unsorted inside a contig) as numpy arrays, their contig offsets,
    and the queries as device tensors: starts, ends, contig ids (None with one contig)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dt = torch.int64 if case["bits"] == 64 else torch.int32
    lens = contig_lengths(case)
    cnt = per_contig(case["n"], lens)
    seg = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int64)
    contig = torch.repeat_interleave(torch.arange(len(lens), device="cuda"), torch.from_numpy(cnt).cuda())
    s = starts(gen, case, case["n"], contig)
    e = s + lengths(gen, case["n"], case["kind"], False) - 1
    intervals = (s.to(dt).cpu().numpy(), e.to(dt).cpu().numpy(), seg)
    del s, e, contig
    nq = case["nq"]
    w = torch.tensor(lens, dtype=torch.float64, device="cuda")
    cdf = torch.cumsum(w, 0) / w.sum()
    qc = torch.searchsorted(cdf, torch.rand(nq, generator=gen, device="cuda", dtype=torch.float64))
    qc = qc.clamp_(0, len(lens) - 1)
    qs = starts(gen, case, nq, qc)
    ql = lengths(gen, nq, case["kind"], True)
    if case["ordered"]:
        at = torch.argsort(qc * (1 << 33) + qs)
        qc, qs = qc[at], qs[at]
    qe = qs + ql - 1
    return intervals, qs.to(dt), qe.to(dt), (qc.to(torch.int32) if len(lens) > 1 else None)


def capacity(case):
    """Slots of the result buffers: the expected hits and what a batch of this size may have above
    them (few long intervals, few long queries)."""
    hits = expected_hits(case)
    hits *= 1.02 + 8 / math.sqrt(0.01 * case["n"] + 1) + 15 / math.sqrt(case["nq"])
    return int(hits) + 4096 + (case["nq"] if case["op"] == "difference" else 0)


def built(case, intervals):
    from superintervals_gb300 import GpuIndex
    idx = GpuIndex(case["bits"])
    idx.add_arrays(intervals[0], intervals[1], None, seg=intervals[2])
    if case["op"] == "upper_bound":
        from superintervals_gb300.interval_map import UB_LEARNED
        idx.set_upper_bound(UB_LEARNED)
    idx.build()
    return idx


def prepare(case, seed):
    intervals, qs, qe, qc = make_inputs(case, seed)
    if case["op"] == "build":
        return {"case": case, "intervals": intervals}
    op, nq = case["op"], case["nq"]
    st = {"case": case, "total": C.c_size_t(0), "cap": capacity(case), "q": [qs, qe, qc]}
    where = {"device": "cpu", "pin_memory": True} if op in ("host_search", "lookup") else {"device": "cuda"}
    if op == "host_search":  # a server's pinned buffers
        st["q"] = [None if a is None else a.cpu().pin_memory() for a in (qs, qe, qc)]
    elif op == "lookup":
        st["q"] = [None if a is None else a.cpu().numpy() for a in (qs, qe, qc)]
    # the caller's result buffers: offsets (or one value a query), and the fields of every hit or piece
    coord, i32, i64 = qs.dtype, torch.int32, torch.int64
    per_query = {"count": [i32], "coverage": [i64, coord], "upper_bound": [i32]}.get(op)
    per_hit = {"keys": [coord, coord, i32], "intersect": [coord, coord, i32], "difference": [coord, coord]}.get(op, [i32])
    if per_query:
        st["out"] = [torch.zeros(nq, dtype=t, **where) for t in per_query]
    else:
        st["out"] = [torch.zeros(nq + 1, dtype=i64, **where)]
        st["out"] += [torch.zeros(st["cap"], dtype=t, **where) for t in per_hit]
    torch.cuda.empty_cache()  # the index's own allocations come from the same card
    st["idx"] = built(case, intervals)
    return st


# ---------------------------------------------------------------- one pass
def ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def run(st):
    from superintervals_gb300._capi import check
    from superintervals_gb300.interval_map import ORDER_DESC, ORDER_IDXS_CPP, UB_LEARNED
    case = st["case"]
    op = case["op"]
    if op == "build":
        from superintervals_gb300 import GpuIndex
        s, e, seg = st["intervals"]
        idx = GpuIndex(case["bits"])
        idx.add_arrays(s, e, None, seg=seg)
        idx.build()
        arrays = idx.arrays()
        idx.close()
        return arrays
    idx = st["idx"]
    if op == "lookup":
        off, hits = idx.search(*st["q"])
        st["out"][0].numpy()[:] = off
        st["out"][1].numpy()[:len(hits)] = hits
        return st["out"]
    lib, h, nq, total = idx.lib, idx.h, case["nq"], st["total"]
    qs, qe, qc = (ptr(t) for t in st["q"])
    out = [ptr(t) for t in st["out"]]
    if op == "host_search":
        check(lib.searchBatchIntoGpu(h, qs, qe, qc, nq, ORDER_IDXS_CPP, 0, out[0], out[1], st["cap"], C.byref(total)))
    elif op == "search":
        check(lib.searchDeviceGpu(h, qs, qe, qc, nq, ORDER_IDXS_CPP, 0, out[0], out[1], st["cap"], C.byref(total), None))
    elif op == "values":
        check(lib.searchDeviceGpu(h, qs, qe, qc, nq, ORDER_DESC, 1, out[0], out[1], st["cap"], C.byref(total), None))
    elif op == "keys":
        check(lib.searchKeysDeviceGpu(h, qs, qe, qc, nq, ORDER_DESC, *out, st["cap"], C.byref(total), None))
    elif op == "intersect":
        check(lib.intersectDeviceGpu(h, qs, qe, qc, nq, ORDER_IDXS_CPP, *out, st["cap"], C.byref(total), None))
    elif op == "difference":
        check(lib.differenceDeviceGpu(h, qs, qe, qc, nq, *out, st["cap"], C.byref(total), None))
    elif op == "count":
        check(lib.countOverlapsDeviceGpu(h, qs, qe, qc, nq, out[0], None))
    elif op == "coverage":
        check(lib.coverageDeviceGpu(h, qs, qe, qc, nq, *out, None))
    elif op == "upper_bound":
        check(lib.upperBoundDeviceGpu(h, qe, qc, nq, UB_LEARNED, out[0], None))
    return st["out"]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: each query read once (start, end and, with several contigs, contig id), the index
    fields that its answer rests on (at most the whole array; a query needs one entry of each at
    least), and each result written once.  No floating-point work."""
    s, n, nq = case["bits"] // 8, case["n"], case["nq"]
    hits = expected_hits(case)
    query = nq * (2 * s + (4 if len(contig_lengths(case)) > 1 else 0))
    index = 2 * s * min(n, nq)
    out = {
        "search": 8 * nq + 4 * hits, "values": 8 * nq + 4 * hits, "host_search": 8 * nq + 4 * hits,
        "lookup": 8 * nq + 4 * hits,
        "keys": 8 * nq + (2 * s + 4) * hits, "intersect": 8 * nq + (2 * s + 4) * hits,
        "difference": 8 * nq + 2 * s * nq, "count": 4 * nq, "coverage": (8 + s) * nq, "upper_bound": 4 * nq,
    }
    if case["op"] == "build":
        return {"bytes": n * (2 * s) + n * (2 * s + 4 + 8), "flops": 0}
    if case["op"] == "upper_bound":
        query, index = nq * s, s * min(n, nq)
    return {"bytes": query + index + out[case["op"]], "flops": 0}
