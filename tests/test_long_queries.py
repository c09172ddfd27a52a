"""Queries longer than a tile's (emit_alone): run lengths on both sides of what a round writes."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from superintervals_gb300 import interval_map
    return interval_map


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
