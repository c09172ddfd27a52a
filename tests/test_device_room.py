"""The rank grids and the gaps are optional: under a device budget a build and every call fit where the
required tables and workspaces do, with the answers of an index that has them."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api():
    from superintervals_gb300 import interval_map
    return interval_map


@pytest.fixture
def budget(api):
    lib = api._capi.load()
    yield lambda b: lib.setDeviceBudgetGpu(int(b))
    lib.setDeviceBudgetGpu(0)


def _intervals(n, bits, contigs, in_order):
    rng = np.random.default_rng(n)
    s = rng.integers(0, 10 * n, n)
    seg = np.linspace(0, n, contigs + 1).astype(np.int64)
    if in_order:
        for g in range(contigs):
            s[seg[g]:seg[g + 1]].sort()
    dt = np.int32 if bits == 32 else np.int64
    return s.astype(dt), (s + rng.integers(0, 60, n) * (not in_order) + 5).astype(dt), seg


# bytes an interval that building took before there were grids
@pytest.mark.parametrize("bits,in_order,contigs,per_interval", [
    (32, False, 1, 56.7), (32, False, 24, 64.7), (32, True, 1, 52.7), (32, True, 24, 60.7),
    (64, False, 1, 88.9), (64, False, 24, 96.9), (64, True, 1, 80.9), (64, True, 24, 88.9)])
def test_build_in_the_room_of_the_required(api, budget, bits, in_order, contigs, per_interval):
    n = 1_000_000
    s, e, seg = _intervals(n, bits, contigs, in_order)
    idx = api.GpuIndex(bits)
    idx.add_arrays(s, e, seg=seg)
    budget(idx.lib.deviceBytesInUseGpu() + per_interval * n)
    idx.build()
    budget(0)
    ss, ee, dd, br = idx.arrays()
    free = api.GpuIndex(bits)
    free.add_arrays(s, e, seg=seg)
    free.build()
    for a, b in zip((ss, ee, dd, br), free.arrays()):
        assert np.array_equal(a, b)
    qs, qe, qc = s[::50], e[::50], np.repeat(np.arange(contigs), np.diff(seg))[::50].astype(np.int32)
    assert np.array_equal(idx.count(qs, qe, qc), free.count(qs, qe, qc))
    idx.close()
    free.close()


def _calls(api, s, e, qc):
    """Name -> a call of an index; each returns arrays."""
    qs, qe = s, e

    def device(idx):
        dev, lib, nq = [], idx.lib, len(qe)
        for a in (qe, qc, np.zeros(nq, np.int32)):
            p = C.c_void_p()
            api.check(lib.deviceMallocGpu(C.byref(p), a.nbytes))
            api.check(lib.memcpyGpu(p, C.c_void_p(a.ctypes.data), a.nbytes, idx.stream))
            dev.append(p)
        got = np.empty(nq, np.int32)
        st = lib.upperBoundDeviceGpu(idx.h, dev[0], dev[1], nq, 0, dev[2], None)
        api.check(lib.memcpyGpu(C.c_void_p(got.ctypes.data), dev[2], got.nbytes, idx.stream))
        api.check(lib.streamSynchronizeGpu(idx.stream))
        for p in dev:
            lib.deviceFreeGpu(p)
        api.check(st)
        return [got]

    return {"count": lambda i: [i.count(qs, qe, qc)], "search": lambda i: i.search(qs, qe, qc),
            "one_search": lambda i: i.search(qs[:1], qe[:1], qc[:1]),
            "values": lambda i: i.search(qs, qe, qc, order=1, values=True),
            "any": lambda i: [i.has_overlaps(qs, qe, qc)], "upper_bound": device,
            "provider": lambda i: (i.set_upper_bound(api.UB_LEARNED), [i.count(qs, qe, qc)])[1],
            "keys": lambda i: i.search_keys(qs, qe, qc, with_data=True), "intersect": lambda i: i.intersect(qs, qe, qc),
            "difference": lambda i: i.difference(qs - 7, qe + 7, qc), "coverage": lambda i: i.coverage(qs, qe, qc)}


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("first", ["count", "search", "one_search", "values", "any", "provider"])
def test_calls_in_the_room_of_the_required(api, budget, first, bits):
    """A first call with the room that an index without the tables and this call's workspace need; then
    every call without the tables."""
    n = 2_000_000
    s, e, seg = _intervals(n, bits, 3, False)
    qc = np.repeat(np.arange(3), np.diff(seg))[::100].astype(np.int32)
    calls = _calls(api, s[::100], e[::100], qc)
    free = api.GpuIndex(bits)
    free.add_arrays(s, e, seg=seg)
    free.build()
    want = {k: [np.array(a) for a in f(free)] for k, f in calls.items()}
    free.close()
    idx = api.GpuIndex(bits)
    others = idx.lib.deviceBytesInUseGpu()
    idx.add_arrays(s, e, seg=seg)
    idx.build()
    budget(others + (24 if bits == 32 else 36) * n + (8 << 20))
    for k in [first] + list(calls):
        got = calls[k](idx)
        assert all(np.array_equal(a, b) for a, b in zip(got, want[k])), k
        budget(0)
    idx.close()


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("call", ["difference", "coverage", "keys", "intersect"])
def test_calls_at_every_budget(api, budget, call, bits):
    """Between no room at all and room for everything a call is refused for want of it or exact, and
    what it could not finish holds nothing."""
    n = 500_000
    s, e, seg = _intervals(n, bits, 3, False)
    qc = np.repeat(np.arange(3), np.diff(seg))[::50].astype(np.int32)
    run = _calls(api, s[::50], e[::50], qc)[call]
    want, served = None, 0
    for room in [None] + [k << 20 for k in range(-8, 40, 3)]:
        idx = api.GpuIndex(bits)
        idx.add_arrays(s, e, seg=seg)
        idx.build()
        if room is not None:
            budget(idx.lib.deviceBytesInUseGpu() + room)
        try:
            got = [np.array(a) for a in run(idx)]
        except api.SIError as ex:
            assert room is not None and ex.status == api._capi.SI_ERR_OOM
            budget(0)
            got = [np.array(a) for a in run(idx)]
        else:
            served += 1
        budget(0)
        want = want or got
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), room
        idx.close()
    assert served > 2
