"""Counts, upper bounds and coverage from the rank grid against numpy ranks, at the shapes where the
grid's buckets can go wrong: crowded and one-coordinate buckets, huge gaps, type extremes, empty and
one-interval contigs, keys at and beside every bucket edge, queries with start > end."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from superintervals_gb300 import interval_map
    return interval_map


def _starts(rng, kind, n, dt):
    info = np.iinfo(dt)
    if kind == "uniform":
        return rng.integers(0, 50 * n + 1, n)
    if kind == "duplicates":                    # one-coordinate buckets of many equal keys
        return rng.choice(np.array([5, 6, 900, 70_000]), n)
    if kind == "gap":                           # nearly all keys in one bucket, one far away
        s = rng.integers(0, 200, n)
        s[0] = info.max - 10
        return s
    if kind == "extremes":                      # the whole coordinate range
        s = rng.integers(info.min // 2, info.max // 2, n)
        s[: n // 3] = info.min
        s[n // 3: n // 2] = info.max
        return s
    s = rng.integers(0, 10_000_000, n)          # "clustered": sub-tables with entries left to search
    hot = rng.random(n) < 0.8
    s[hot] = 4_000_000 + np.rint(rng.standard_normal(int(hot.sum())) * 3000).astype(np.int64)
    return s


def _case(kind, n, dt, seed):
    rng = np.random.default_rng(seed)
    info = np.iinfo(dt)
    s = _starts(rng, kind, n, dt).astype(np.int64)
    room = np.array([info.max - int(x) for x in s], dtype=np.float64)
    ln = np.minimum(rng.integers(0, 3000, n), room).astype(np.int64)
    e = s + ln
    # contigs: an empty one first, one interval, the rest split in two, an empty one last
    cut = sorted({0, min(1, n), (n + 1) // 2, n})
    seg = np.array([0] + cut + [n], dtype=np.int64)
    G = len(seg) - 1
    # queries on, beside and between the keys, in every contig, some with start > end
    near = rng.choice(np.concatenate([s, e]), 3000)
    qs = np.array([min(max(int(v) + int(d), info.min), info.max) for v, d in zip(near, rng.integers(-2, 3, 3000))])
    qe = np.array([min(int(v) + int(d), info.max) for v, d in zip(qs, rng.choice([0, 1, 40, 5000], 3000))])
    qe[:50], qs[:50] = qs[:50].copy(), qe[:50].copy()
    qs[50:60], qe[50:60] = info.min, info.max
    qc = rng.integers(0, G, 3000)
    return s.astype(dt), e.astype(dt), seg, qs.astype(dt), qe.astype(dt), qc.astype(np.int32)


def _expected(s, e, seg, qs, qe, qc):
    ub = np.full(len(qs), -1, np.int64)
    cnt = np.zeros(len(qs), np.int64)
    for g in range(len(seg) - 1):
        a, b = s[seg[g]:seg[g + 1]], e[seg[g]:seg[g + 1]]
        sel = np.flatnonzero(qc == g)
        ub[sel] = np.searchsorted(np.sort(a), qe[sel], side="right") - 1
        cnt[sel] = [int(((a <= y) & (b >= x)).sum()) for x, y in zip(qs[sel], qe[sel])]
    return ub, cnt


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("n", [1, 2, 7, 33, 1000, 4097])
@pytest.mark.parametrize("kind", ["uniform", "duplicates", "gap", "extremes", "clustered"])
def test_ranks_match_numpy(api, kind, n, dt):
    s, e, seg, qs, qe, qc = _case(kind, n, dt, seed=n)
    ub, cnt = _expected(s, e, seg, qs, qe, qc)
    idx = api.GpuIndex(np.dtype(dt).itemsize * 8)
    idx.add_arrays(s, e, seg=seg)
    idx.build()
    assert np.array_equal(idx.count(qs, qe, qc), cnt)
    lib, nq = idx.lib, len(qs)
    d = []
    for a in (qe, qc, np.zeros(nq, np.int32)):
        p = C.c_void_p()
        api.check(lib.deviceMallocGpu(C.byref(p), a.nbytes))
        api.check(lib.memcpyGpu(p, C.c_void_p(a.ctypes.data), a.nbytes, idx.stream))
        d.append(p)
    api.check(lib.upperBoundDeviceGpu(idx.h, d[0], d[1], nq, 0, d[2], None))
    got = np.empty(nq, np.int32)
    api.check(lib.memcpyGpu(C.c_void_p(got.ctypes.data), d[2], got.nbytes, idx.stream))
    api.check(lib.streamSynchronizeGpu(idx.stream))
    assert np.array_equal(got, ub)
    for p in d:
        lib.deviceFreeGpu(p)
    # coverage, with and without queries that have start > end, in the wrapping coordinate type
    for sel in (np.flatnonzero(qs <= qe)[:400], np.arange(400)):
        c2, cov = idx.coverage(qs[sel], qe[sel], qc[sel])
        assert np.array_equal(c2, cnt[sel])
        for k, i in enumerate(sel[::13]):
            a, b = (v[seg[qc[i]]:seg[qc[i] + 1]].astype(object) for v in (s, e))
            hit = [(x, y) for x, y in zip(a, b) if x <= int(qe[i]) and y >= int(qs[i])]
            want = sum(min(int(y), int(qe[i])) - max(int(x), int(qs[i])) for x, y in hit)
            bits = np.dtype(dt).itemsize * 8
            want = (want + (1 << (bits - 1))) % (1 << bits) - (1 << (bits - 1))
            assert int(cov[13 * k]) == want
    idx.close()


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("width", [1, 2, 6, 7, 8, 15, 16, 17, 24])
def test_offsets_inside_buckets(api, width, dt):
    """Buckets of 2^width coordinates with 0 to 40 entries each, at every alignment in the 8-entry
    blocks, keys on both bucket edges; widths on both sides of what a 7-bit code and a 16-bit offset
    hold."""
    if width > 17 and dt is np.int32:
        pytest.skip("1024 buckets of 2^24 pass the 32-bit range")
    rng = np.random.default_rng(width)
    n, nb = 4096, 1024
    first = np.sort(np.repeat(np.arange(nb), rng.integers(0, 41, nb))[:n - 2])
    first = np.concatenate([first, np.full(n - 2 - len(first), nb // 2)]).astype(np.int64)
    inside = rng.choice(np.array([0, 1, (1 << width) // 2, (1 << width) - 1]), n - 2)
    s = np.concatenate([[0, (nb << width) - 1], (first << width) + np.minimum(inside, (1 << width) - 1)]) - 77
    e = s + rng.integers(0, 3 << width, n)
    qe = np.concatenate([s, s - 1, s + 1])
    qs = qe - rng.integers(0, 2 << width, len(qe))
    cnt = np.searchsorted(np.sort(s), qe, side="right") - np.searchsorted(np.sort(e), qs, side="left")
    idx = api.GpuIndex(np.dtype(dt).itemsize * 8)
    idx.add_arrays(s.astype(dt), e.astype(dt))
    idx.build()
    assert np.array_equal(idx.count(qs.astype(dt), qe.astype(dt)), cnt)
    idx.close()


def _uncovered(s, e, lo, hi):
    """Stretches of [lo, hi] that no interval [s, e] covers, as exact Python ints."""
    out, cur = [], lo
    for a, b in sorted(zip(s.tolist(), e.tolist())):
        if a > hi or b < lo:
            continue
        if a > cur:
            out.append((cur, a - 1))
        cur = max(cur, b + 1)
    if cur <= hi:
        out.append((cur, hi))
    return out


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("n", [1, 2, 7, 33, 1000, 4097])
@pytest.mark.parametrize("kind", ["uniform", "duplicates", "gap", "extremes", "clustered"])
def test_difference_from_gaps(api, kind, n, dt):
    s, e, seg, qs, qe, qc = _case(kind, n, dt, seed=n + 1)
    e = s + np.minimum(e - s, 100).astype(dt)                # leave gaps between the intervals
    sel = np.concatenate([np.arange(120), np.arange(2500, 2700)])
    qs, qe, qc = qs[sel], qe[sel], qc[sel]
    idx = api.GpuIndex(np.dtype(dt).itemsize * 8)
    idx.add_arrays(s, e, seg=seg)
    idx.build()
    off, ps, pe = idx.difference(qs, qe, qc)
    for i in range(len(qs)):
        a, b = (v[seg[qc[i]]:seg[qc[i] + 1]] for v in (s, e))
        want = _uncovered(a, b, int(qs[i]), int(qe[i])) if qs[i] <= qe[i] else []
        got = list(zip(ps[off[i]:off[i + 1]].tolist(), pe[off[i]:off[i + 1]].tolist()))
        assert got == want
    idx.set_path(api.PATH_PLAIN)                             # the hit-list sweep
    off2, ps2, pe2 = idx.difference(qs, qe, qc)
    assert np.array_equal(off, off2) and np.array_equal(ps, ps2) and np.array_equal(pe, pe2)
    idx.close()


def test_count_paths_agree(api):
    s, e, seg, qs, qe, qc = _case("uniform", 4097, np.int32, seed=5)
    _, cnt = _expected(s, e, seg, qs, qe, qc)
    idx = api.GpuIndex(32)
    idx.add_arrays(s, e, seg=seg)
    idx.build()
    assert np.array_equal(idx.count(qs, qe, qc), cnt)
    for path in (api.PATH_PLAIN, api.PATH_BATCHED):
        idx.set_path(path)
        assert np.array_equal(idx.count(qs, qe, qc), cnt)
    idx.close()


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("nq", [1, 2, 31, 33, 257, 2431, 2433, 4865, 155_649])
def test_few_queries_with_many_gaps(api, nq, bits):
    """Stretches of pieces shared by 64 warps down to one each, empty queries among them."""
    dt = np.int32 if bits == 32 else np.int64
    n = 5000 if nq > 300 else 40_000
    s = (np.arange(n) * 10).astype(dt)                        # a gap of 4 behind each interval
    rng = np.random.default_rng(nq)
    lo = np.sort(rng.integers(0, n - 1, (2, nq)), axis=0)
    if nq > 3000:
        lo[1] = np.minimum(lo[0] + rng.integers(0, 40, nq), n - 1)
    qs, qe = (lo[0] * 10 + 7).astype(dt), (lo[1] * 10 + 8).astype(dt)
    none = rng.random(nq) < 0.2
    qs[none], qe[none] = lo[0][none] * 10, lo[0][none] * 10 + 5
    idx = api.GpuIndex(bits)
    idx.add_arrays(s, s + 5)
    idx.build()
    off, ps, pe = idx.difference(qs, qe)
    cnt = np.where(none, 0, lo[1] - lo[0] + 1)
    want_off = np.concatenate([[0], np.cumsum(cnt)])
    assert np.array_equal(off, want_off)
    gap = np.repeat(lo[0], cnt) + np.arange(want_off[-1]) - np.repeat(want_off[:-1], cnt)
    assert np.array_equal(ps, np.maximum(gap * 10 + 6, np.repeat(qs, cnt)))
    assert np.array_equal(pe, np.minimum(gap * 10 + 9, np.repeat(qe, cnt)))
    idx.close()


def test_few_long_differences_take_the_device(api):
    """300 differences of 20 k pieces each: 4.2 ms by ten warps."""
    import time

    n, nq = 20_000, 300
    s = np.arange(n, dtype=np.int32) * 10
    idx = api.GpuIndex(32)
    idx.add_arrays(s, s + 5)
    idx.build()
    lib, cap, best = idx.lib, n * nq + 1000, 1.0
    bufs = [C.c_void_p() for _ in range(5)]
    for b, size in zip(bufs, (4 * nq, 4 * nq, 8 * (nq + 1), 4 * cap, 4 * cap)):
        api.check(lib.deviceMallocGpu(C.byref(b), size))
    ends = np.full(nq, 10 * n, np.int32)
    for b, a in zip(bufs, (np.zeros(nq, np.int32), ends)):
        api.check(lib.memcpyGpu(b, C.c_void_p(a.ctypes.data), a.nbytes, idx.stream))
    total = C.c_size_t(0)
    for _ in range(6):
        t = time.perf_counter()
        api.check(lib.differenceDeviceGpu(idx.h, bufs[0], bufs[1], None, nq, bufs[2], bufs[3], bufs[4], cap,
                                          C.byref(total), None))
        best = min(best, time.perf_counter() - t)
    assert total.value == n * nq and best < 0.0015
    for b in bufs:
        lib.deviceFreeGpu(b)
    idx.close()


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("n", [25, 300, 5000, 300_000])
@pytest.mark.parametrize("shape", ["outlier", "low", "two", "ladder", "steps", "equal"])
def test_crowded_buckets(api, shape, n, dt):
    """Buckets with their own tables over their entries' range: nearly all entries in one bucket, a cluster
    at each end of a bucket, clusters of every width, long stretches of one table between two entries, and
    buckets of equal entries."""
    info = np.iinfo(dt)
    rng = np.random.default_rng(n)
    top = int(info.max) - 3000
    s = rng.integers(0, 40 * n, n)
    if shape == "outlier":
        s[0] = top
    elif shape == "low":
        s[0] = info.min + 5
    elif shape == "two":
        s[: n // 2] += top // 2
    elif shape == "ladder":                                   # a cluster around every power of two
        s = (1 << rng.integers(0, int(info.bits) - 2, n)) + rng.integers(0, 50, n)
    elif shape == "steps":                                    # pairs far apart inside a crowded bucket
        s = np.sort(rng.integers(0, 30, n)) * (top // 64) + rng.choice([0, 1, 9_000_000], n)
        s[0] = info.min // 2
    else:
        s = rng.choice([7, 8, 5000, top // 3], n)
    e = s + rng.integers(0, 90, n)
    s, e = s.astype(dt), e.astype(dt)
    near = rng.choice(np.concatenate([s, e]), 20_000).astype(object)
    qs = np.array([min(max(v + d, int(info.min)), int(info.max) - 200) for v, d in
                   zip(near, rng.integers(-3, 4, len(near)).tolist())]).astype(dt)
    qe = qs + rng.choice(np.array([0, 1, 100], dt), len(qs))
    qs[:100] = info.min
    qe[100:200] = info.max
    cnt = np.searchsorted(np.sort(s), qe, side="right") - np.searchsorted(np.sort(e), qs, side="left")
    idx = api.GpuIndex(np.dtype(dt).itemsize * 8)
    idx.add_arrays(s, e)
    idx.build()
    assert np.array_equal(idx.count(qs, qe), cnt)
    got = idx.coverage(qs, qe)
    idx.set_path(api.PATH_BATCHED)
    for a, b in zip(got, idx.coverage(qs, qe)):
        assert np.array_equal(a, b)
    idx.close()


def test_one_outlying_coordinate_costs_little(api):
    """5 M counts over 5 M intervals with 64-bit coordinates: 6.7 times as long with one interval far behind
    the others, which then all lay in one bucket and one sub-bucket; 1.9 times now."""
    import time

    rng = np.random.default_rng(2)
    n, ms = 5_000_000, []
    for far in (False, True):
        s = rng.integers(0, 249_000_000, n)
        if far:
            s[0] = 1 << 62
        idx = api.GpuIndex(64)
        idx.add_arrays(s, s + 800)
        idx.build()
        qs = rng.integers(0, 249_000_000, n)
        lib, bufs = idx.lib, [C.c_void_p() for _ in range(3)]
        for b, a in zip(bufs, (qs, qs + 800, np.zeros(n, np.uint32))):
            api.check(lib.deviceMallocGpu(C.byref(b), a.nbytes))
            api.check(lib.memcpyGpu(b, C.c_void_p(a.ctypes.data), a.nbytes, idx.stream))
        best = 1e9
        for _ in range(6):
            api.check(lib.streamSynchronizeGpu(idx.stream))
            t = time.perf_counter()
            api.check(lib.countOverlapsDeviceGpu(idx.h, bufs[0], bufs[1], None, n, bufs[2], None))
            api.check(lib.streamSynchronizeGpu(idx.stream))
            best = min(best, 1e3 * (time.perf_counter() - t))
        ms.append(best)
        for b in bufs:
            lib.deviceFreeGpu(b)
        idx.close()
    assert ms[1] < 3.5 * ms[0]


def _grid_shift(keys):
    """log2 of the bucket width that the grid takes for these ascending keys (k_grid_params)."""
    n, span = len(keys), int(keys[-1]) - int(keys[0])
    at = [int(keys[(n - 1) * k // 64]) for k in range(65)]
    spread = sum(b - a >= span // 256 for a, b in zip(at, at[1:]))
    cap, shift = max(2, n * spread // 64 // 4), 0
    while span >> shift >= cap:
        shift += 1
    return shift


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("width", [0, 1, 6, 7, 8, 9, 15, 16, 17, 20, 33])
def test_bucket_widths(api, width, dt):
    """Starts and ends in buckets of exactly 2^width coordinates, on both sides of what a record's seven-bit
    code and a 16-bit offset hold, with records of all codes (up to 12 entries), counts only (13-19) and
    tables of their own (20 and more), entries on both bucket edges and equal ones among them."""
    if width > 20 and dt is np.int32:
        pytest.skip("1000 buckets of 2^33 pass the 32-bit range")
    rng = np.random.default_rng(width)
    n, nb = 4096, 1000
    per = rng.choice([0, 1, 2, 3, 4, 5, 6, 7, 8, 12], nb, p=[.1, .1, .15, .2, .15, .1, .08, .05, .05, .02])
    per[10::50] = rng.integers(20, 41, len(per[10::50]))
    per[35::50] = rng.integers(13, 20, len(per[35::50]))
    while per.sum() != n:                                     # to exactly n, in buckets of few entries
        k = rng.integers(1, nb - 1)
        if per[k] < 12:
            per[k] = min(max(per[k] + np.sign(n - per.sum()), 0), 11)
    per[0], per[1], per[-2], per[-1] = 1, per[:2].sum() - 1, per[-2:].sum() - 1, 1
    b = np.repeat(np.arange(nb), per)
    w = 1 << width
    inside = rng.integers(0, w, n) if width < 6 else np.where(rng.random(n) < 0.3, rng.choice([0, 1, w // 2, w - 1], n),
                                                               rng.integers(0, w, n))
    inside[0], inside[-1] = 0, w - 1
    s = np.sort((b << width) + inside) - 77
    e = s + 5 * w + 1
    assert _grid_shift(s) == width and _grid_shift(e) == width
    got = np.bincount((s - s[0]) >> width)
    assert (got > 20).any() and ((got >= 13) & (got < 20)).any() and (got == 12).any()
    edges = ((np.arange(nb + 1) << width) - 77)
    qe = np.concatenate([s, s - 1, s + 1, edges, edges - 1, edges + w // 2])
    qs = rng.permutation(np.concatenate([e, e - 1, e + 1, edges + 5 * w + 1, edges + 5 * w, edges + 5 * w + w // 2]))
    qs = np.minimum(qs, qe)
    near = np.arange(len(qe)) % 2 == 0                        # the end's rank from a key of its own
    qs[near] = qe[near] - rng.integers(0, 6 * w, near.sum())
    info = np.iinfo(dt)
    assert s[0] > info.min and e[-1] + w < info.max
    cnt = np.searchsorted(s, qe, side="right") - np.searchsorted(e, qs, side="left")
    idx = api.GpuIndex(np.dtype(dt).itemsize * 8)
    idx.add_arrays(s.astype(dt), e.astype(dt))
    idx.build()
    assert np.array_equal(idx.count(qs.astype(dt), qe.astype(dt)), cnt)
    got = idx.coverage(qs.astype(dt), qe.astype(dt))
    idx.set_path(api.PATH_PLAIN)
    for x, y in zip(got, idx.coverage(qs.astype(dt), qe.astype(dt))):
        assert np.array_equal(x, y)
    idx.close()
