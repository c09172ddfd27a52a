"""Queries longer than a tile's (emit_alone): run lengths on both sides of what a round writes, and windows
of the long-interval list that one contig-long interval makes as long as the list."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from superintervals_gb300 import interval_map
    return interval_map


@pytest.fixture(scope="module")
def oracle():
    from oracle.oracle import Oracle
    return Oracle()


@pytest.mark.parametrize("bits", [32, 64])
def test_run_lengths(api, bits):
    dt = np.int32 if bits == 32 else np.int64
    n = 3000
    s = (np.arange(n) * 1000).astype(dt)
    e = s + 1500                                             # each also reaches into the next one
    data = np.random.default_rng(bits).integers(-9, 9, n).astype(np.int32)
    runs = np.array([1, 2, 31, 32, 33, 95, 96, 97, 127, 128, 129, 160, 255, 256, 257, 511, 513, 1000, 2900])
    first = np.random.default_rng(bits).integers(0, n - runs)
    qs, qe = (first * 1000).astype(dt), ((first + runs - 1) * 1000 + 10).astype(dt)
    idx = api.GpuIndex(bits)
    idx.add_arrays(s, e, data)
    idx.build()
    idx.set_path(api.PATH_BATCHED)
    api.check(idx.lib.setBatchedParamsGpu(idx.h, 0, 0, 1, -1))  # every query is a long one
    for order in (api.ORDER_IDXS_CPP, api.ORDER_DESC):
        want = [np.flatnonzero((s <= b) & (e >= a))[::-1 if order == api.ORDER_DESC else 1] for a, b in zip(qs, qe)]
        off = np.concatenate([[0], np.cumsum([len(w) for w in want])])
        want = np.concatenate(want)
        owner = np.repeat(np.arange(len(runs)), np.diff(off))
        got_off, got = idx.search(qs, qe, order=order)
        assert np.array_equal(got_off, off) and np.array_equal(got, want)
        got_off, got = idx.search(qs, qe, order=order, values=True)
        assert np.array_equal(got_off, off) and np.array_equal(got, data[want])
        got_off, ps, pe, ph = idx.intersect(qs, qe, order=order)
        assert np.array_equal(got_off, off) and np.array_equal(ph, want)
        assert np.array_equal(ps, np.maximum(s[want], qs[owner])) and np.array_equal(pe, np.minimum(e[want], qe[owner]))
    idx.close()


class _Device:
    """A batch in device memory, with room for `cap` results; `ms` is the shortest of a few searches."""

    def __init__(self, api, idx, qs, qe, cap):
        self.api, self.idx, self.cap, self.nq = api, idx, cap, len(qs)
        self.bufs = [C.c_void_p() for _ in range(4)]
        for b, size in zip(self.bufs, (qs.nbytes, qe.nbytes, 8 * (len(qs) + 1), 4 * cap)):
            api.check(idx.lib.deviceMallocGpu(C.byref(b), size))
        for b, a in zip(self.bufs, (qs, qe)):
            api.check(idx.lib.memcpyGpu(b, C.c_void_p(a.ctypes.data), a.nbytes, idx.stream))

    def ms(self, values):
        total, best = C.c_size_t(0), 1e9
        for _ in range(6):
            t = time.perf_counter()
            self.api.check(self.idx.lib.searchDeviceGpu(self.idx.h, self.bufs[0], self.bufs[1], None, self.nq,
                                                        self.api.ORDER_DESC, values, self.bufs[2], self.bufs[3],
                                                        self.cap, C.byref(total), None))
            best = min(best, 1e3 * (time.perf_counter() - t))
        return best

    def close(self):
        for b in self.bufs:
            self.idx.lib.deviceFreeGpu(b)


def test_payloads_of_a_long_run_cost_little_more_than_positions(api):
    """Ten queries over 2 M intervals, a warp each: payloads took 15 times the positions' time with a wait
    behind every round of 32, three times with several rounds read at once."""
    n = 2_000_000
    s = np.arange(n, dtype=np.int32) * 100
    idx = api.GpuIndex(32)
    idx.add_arrays(s, s + 150)
    idx.build()
    d = _Device(api, idx, np.zeros(10, np.int32), np.full(10, 100 * n, np.int32), 10 * n + 100)
    assert d.ms(1) < 7 * d.ms(0)
    d.close()
    idx.close()


def _reads(n, nq, span, far, rng, whole):
    """A tenth of the intervals and of the queries 10-50 kb, the others 150; `whole`: one interval over
    everything."""
    def lengths(k):
        return np.where(rng.random(k) < far, rng.integers(10_000, 50_000, k), 150)
    s, qs = rng.integers(0, span, n), rng.integers(0, span, nq)
    e, qe = s + lengths(n), qs + lengths(nq)
    if whole:
        s[0], e[0] = 0, span
    return s, e, qs, qe


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("span", [3_000_000, 60_000_000, 1_500_000_000])
def test_one_interval_over_everything(api, oracle, span, bits):
    dt = np.int32 if bits == 32 else np.int64
    rng = np.random.default_rng(span)
    s, e, qs, qe = (a.astype(dt) for a in _reads(30_000, 6_000, span, 0.3, rng, True))
    data = rng.integers(-5, 1 << 30, len(s)).astype(np.int32)
    m = oracle.build(s, e, data, seg=np.array([0, len(s)]))
    idx = api.GpuIndex(bits)
    idx.add_arrays(s, e, data)
    idx.build()
    ss, se, sd, _ = idx.arrays()
    for path in (api.PATH_AUTO, api.PATH_BATCHED):
        idx.set_path(path)
        for order in (0, 1):
            want_off, want = oracle.search_batch(m, qs, qe, None, order=order, nthreads=8)
            off, out = idx.search(qs, qe, order=order)
            assert np.array_equal(off, want_off) and np.array_equal(out, want)
            off, out = idx.search(qs, qe, order=order, values=True)
            assert np.array_equal(off, want_off) and np.array_equal(out, sd[want])
            owner = np.repeat(np.arange(len(qs)), np.diff(want_off))
            off, ps, pe, ph = idx.intersect(qs, qe, order=order)
            assert np.array_equal(off, want_off) and np.array_equal(ph, want)
            assert np.array_equal(ps, np.maximum(ss[want], qs[owner]))
            assert np.array_equal(pe, np.minimum(se[want], qe[owner]))
    idx.close()


def test_one_interval_over_everything_costs_little(api):
    """1 M reads against 1 M: with one contig-long interval every long query's window was the whole list of
    long intervals before it, and the call took 6.8 times as long; 1.3 times now."""
    ms = []
    for whole in (False, True):
        s, e, qs, qe = (a.astype(np.int32) for a in _reads(1_000_000, 1_000_000, 249_000_000, 0.1,
                                                           np.random.default_rng(3), whole))
        idx = api.GpuIndex(32)
        idx.add_arrays(s, e)
        idx.build()
        d = _Device(api, idx, qs, qe, 40_000_000)
        ms.append(d.ms(1))
        d.close()
        idx.close()
    assert ms[1] < 2.5 * ms[0]
