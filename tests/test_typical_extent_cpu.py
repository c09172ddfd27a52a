"""The extent that an index's mean density is taken over (typical_extent in si_build.cu), from the function's
own text on the CPU: first to last start, except for what outlying starts add."""
import subprocess

import numpy as np
import pytest

from test_tile_gather_cpu import device_function

MAIN = r"""
#include <cstdint>
#include <cstdio>
#include <vector>
#define __device__
%s
template <typename S> void run() {
    int64_t n;
    if (scanf("%%ld", &n) != 1) return;
    std::vector<S> s(n);
    for (auto& x : s) { long v; if (scanf("%%ld", &v) != 1) return; x = (S)v; }
    printf("%%llu\n", typical_extent<S>(s.data(), n));
}
int main(int argc, char** argv) { argv[1][0] == '4' ? run<int32_t>() : run<int64_t>(); }
"""


@pytest.fixture(scope="module")
def extent(tmp_path_factory):
    d = tmp_path_factory.mktemp("extent")
    (d / "x.cpp").write_text(MAIN % device_function("typical_extent", "si_build.cu"))
    subprocess.run(["g++", "-O1", "-std=c++17", str(d / "x.cpp"), "-o", str(d / "x")], check=True)

    def call(s):
        text = f"{len(s)} " + " ".join(map(str, s.tolist()))
        r = subprocess.run([str(d / "x"), str(s.dtype.itemsize)], input=text, capture_output=True, text=True, check=True)
        return int(r.stdout)
    return call


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 31, 32, 33, 1000, 4099])
def test_even_starts_count_in_full(extent, n, dt):
    s = (np.arange(n) * 37 - 5000).astype(dt)
    assert extent(s) == 37 * (n - 1)


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("low,high", [(1, 0), (0, 1), (3, 3)])
def test_outlying_starts_add_little(extent, low, high, dt):
    n = 5000
    s = np.sort(np.random.default_rng(n).integers(0, 400_000, n)).astype(dt)
    s[:low], s[n - high:] = np.iinfo(dt).min, np.iinfo(dt).max
    assert 300_000 < extent(s) < 800_000


def test_extremes(extent):
    info = np.iinfo(np.int64)
    s = np.linspace(float(info.min), float(info.max), 64).clip(-9.2e18, 9.2e18).astype(np.int64)
    assert extent(s) == int(s[-1]) - int(s[0])                # even: every eighth in full, beyond 63 bits
    assert extent(np.full(100, 7, np.int64)) == 0
    two = np.concatenate([np.arange(500), (1 << 40) + np.arange(500)]).astype(np.int64)
    assert extent(two) < 2000
