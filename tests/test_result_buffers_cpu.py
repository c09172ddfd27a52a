"""The numpy calls' result arrays (GpuIndex.search, search_keys, intersect, difference) over a library that
only reports sizes: what is offered to the first call, and that that is given up before the second one's
arrays are made."""
import tracemalloc

import numpy as np
import pytest

from superintervals_gb300 import _capi
from superintervals_gb300.interval_map import GpuIndex


class _SizesOnly:
    """Stands in for the library: every call has `total` results."""

    def __init__(self, total):
        self.total, self.capacities, self.held = total, [], 0

    def __getattr__(self, name):
        if name == "destroySuperIntervalsGpu":
            return lambda h: None

        def call(*args):
            cap, total = args[-2:]
            total._obj.value = self.total
            self.capacities.append(cap)
            self.held = tracemalloc.get_traced_memory()[1]        # the most since the call before
            tracemalloc.reset_peak()
            return 0 if cap >= self.total else _capi.SI_ERR_CAPACITY
        return call


def _index(total):
    idx = GpuIndex.__new__(GpuIndex)
    idx.h, idx.lib, idx.bits, idx.dtype = 1, _SizesOnly(total), 32, np.int32
    return idx


@pytest.mark.parametrize("call,arrays", [("search_keys", 3), ("intersect", 3), ("difference", 3), ("search", 1)])
@pytest.mark.parametrize("nq", [1, 1000, 1 << 17, (1 << 17) + 1, 1_000_000])
def test_first_call_offers_little_more_than_its_result(call, arrays, nq):
    for total in (nq // 2, nq, 9 * nq + 2000):
        idx = _index(total)
        q = np.zeros(nq, np.int32)
        tracemalloc.start()
        before = tracemalloc.get_traced_memory()[0]
        if call == "search":  # its result is cut to the offsets, which nobody writes here
            try:
                idx.search(q, q)
            except (ValueError, IndexError):
                pass
        else:
            getattr(idx, call)(q, q)
        held = idx.lib.held - before
        tracemalloc.stop()
        first = idx.lib.capacities[0]
        assert first >= nq + 1024 and first <= 4 * nq + 1024
        if arrays > 1 and nq > 1 << 17:
            assert first <= nq + 1024
        assert idx.lib.capacities[1:] == ([total] if total > first else [])
        assert held < 4 * arrays * idx.lib.capacities[-1] + 8 * (nq + 1) + 100_000
