"""The automatic search path's direct emit (2, 8 and 32 lanes per query) and sorted tiles from
upper bounds against the oracle, at the sizes where each starts: batches around the lane limits,
head runs over several chunks, far hits, contig borders inside one key, empty contigs, and the
host-buffer form cut into chunks."""
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


def _intervals(kind, n, rng):
    span = 40 * n
    s = rng.integers(0, span, n)
    if kind == "sparse":
        ln = rng.integers(1, 60, n)
    elif kind == "runs":                       # long head runs: many hits in a row below the bound
        ln = rng.integers(4000, 8000, n)
    else:                                      # "far": a few intervals over everything
        ln = rng.integers(1, 60, n)
        ln[rng.random(n) < 0.002] = span
    if kind == "deep":                         # sections of some 250 long intervals, few of them missed
        ln = rng.integers(1, 60, n)
        deep = rng.random(n) < 0.05
        ln[deep] = rng.integers(100_000, 300_000, int(deep.sum()))
    return s, s + ln - 1, span


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("kind,nq", [(k, q) for k in ("sparse", "runs", "far") for q in (1, 33, 4097, 32769, 262145)]
                         + [("deep", q) for q in (1, 255, 4097, 32769)])
def test_direct_emit_matches_oracle(api, oracle, kind, nq, dt):
    rng = np.random.default_rng(nq)
    n = 20_001
    s, e, span = _intervals(kind, n, rng)
    seg = np.array([0, 0, 7001, 7002, n, n], np.int64)      # empty contigs and a single interval
    G = len(seg) - 1
    qs = rng.integers(-100, span + 100, nq)
    qe = qs + rng.integers(0, 50, nq)
    inv = rng.random(nq) < 0.01                               # start > end
    qs[inv], qe[inv] = qe[inv], qs[inv]
    qc = rng.integers(0, G, nq).astype(np.int32)
    s, e, qs, qe = (a.astype(dt) for a in (s, e, qs, qe))
    d = rng.integers(-5, 1 << 30, n).astype(np.int32)
    m = oracle.build(s, e, d, seg=seg)
    idx = api.GpuIndex(np.dtype(dt).itemsize * 8)
    idx.add_arrays(s, e, d, seg=seg)
    idx.build()
    for path in (api.PATH_AUTO, api.PATH_BATCHED):
        idx.set_path(path)
        for order, values in ((0, False), (1, False), (1, True)):
            want_off, want = oracle.search_batch(m, qs, qe, qc, order=order, nthreads=8)
            off, out = idx.search(qs, qe, qc, order=order, values=values)
            assert np.array_equal(off, want_off)
            if values:
                _, _, data, _ = idx.arrays()
                want = data[want + np.repeat(seg[qc], np.diff(want_off))]
            assert np.array_equal(out, want)
    # the fields written by the emit itself: pieces (none for start > end) and keys
    sorted_s, sorted_e, data, _ = idx.arrays()
    for path in (api.PATH_AUTO, api.PATH_BATCHED):
        idx.set_path(path)
        for order in (0, 1):
            want_off, want = oracle.search_batch(m, qs, qe, qc, order=order, nthreads=8)
            at = want + np.repeat(seg[qc], np.diff(want_off))
            off, ks, ke, kd = idx.search_keys(qs, qe, qc, order=order, with_data=True)
            assert np.array_equal(off, want_off) and np.array_equal(kd, data[at])
            assert np.array_equal(ks, sorted_s[at]) and np.array_equal(ke, sorted_e[at])
            owner = np.repeat(np.arange(nq), np.diff(want_off))
            keep = (qs <= qe)[owner]
            off, ps, pe, ph = idx.intersect(qs, qe, qc, order=order)
            assert np.array_equal(off, np.concatenate([[0], np.cumsum(np.bincount(owner[keep], minlength=nq))]))
            assert np.array_equal(ph, want[keep])
            assert np.array_equal(ps, np.maximum(qs[owner], sorted_s[at])[keep])
            assert np.array_equal(pe, np.minimum(qe[owner], sorted_e[at])[keep])
    idx.set_path(api.PATH_AUTO)
    want_off, want = oracle.search_batch(m, qs, qe, qc, order=0, nthreads=8)
    idx.set_output_budget(1 << 20)                            # host results in chunks
    off, out = idx.search(qs, qe, qc)
    assert np.array_equal(off, want_off) and np.array_equal(out, want)
    idx.close()
