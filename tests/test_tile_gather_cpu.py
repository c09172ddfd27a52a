"""The tiles' block-wide gather (gather_bfs in si_batched.cu) run on the CPU: the function's own text,
compiled with one thread per lane, barriers for the block's and the warps' synchronisation, and every
warp but the first delayed after each block barrier.  Two gathers in a row, as the tile kernels make
them, give the candidates that a direct search finds: a second gather that overwrites what a late
warp has still to read of the first one gives others, or never ends."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "superintervals_gb300", "csrc")

SHIM = r"""
#include <algorithm>
#include <barrier>
#include <chrono>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>
#define __device__
#define __forceinline__ inline
constexpr int kThreads = 256, kWarpsPerCta = 8, kMaxLevels = 8;
constexpr unsigned kFull = 0xffffffffu;
template <typename S> struct Lim;
template <> struct Lim<int32_t> { static constexpr int32_t lo = INT32_MIN, hi = INT32_MAX; };
template <typename S> struct Pyr { const S* ends; const S* m[kMaxLevels]; int H; };
struct Idx { int x; };
thread_local Idx threadIdx;
std::barrier<> block_bar(kThreads);
std::vector<std::unique_ptr<std::barrier<>>> warp_bar;
int lane_val[kThreads];
int __popc(unsigned x) { return __builtin_popcount(x); }
template <typename T> T min(T a, T b) { return a < b ? a : b; }
unsigned above_mask(int lane) { return lane == 31 ? 0u : kFull << (lane + 1); }
void __syncthreads() {
    block_bar.arrive_and_wait();
    if (threadIdx.x >= 32) std::this_thread::sleep_for(std::chrono::milliseconds(20));
}
template <typename F> auto warp_exchange(int v, F read) {
    auto& b = *warp_bar[threadIdx.x / 32];
    lane_val[threadIdx.x] = v;
    b.arrive_and_wait();
    auto r = read(lane_val + (threadIdx.x & ~31));
    b.arrive_and_wait();
    return r;
}
unsigned __ballot_sync(unsigned, bool p) {
    return warp_exchange(p, [](const int* v) {
        unsigned m = 0;
        for (int i = 0; i < 32; ++i) m |= (unsigned)(v[i] != 0) << i;
        return m;
    });
}
int __shfl_up_sync(unsigned, int x, int d) {
    const int lane = threadIdx.x & 31;
    return warp_exchange(x, [=](const int* v) { return lane >= d ? v[lane - d] : v[lane]; });
}
"""

MAIN = r"""
struct Level { std::vector<std::vector<int32_t>> a; Pyr<int32_t> P; };
Level pyramid(std::vector<int32_t> ends) {
    Level L;
    while (ends.size() % 32) ends.push_back(INT32_MIN);
    L.a.push_back(ends);
    while (L.a.back().size() > 32) {
        std::vector<int32_t> up;
        const auto& b = L.a.back();
        for (size_t i = 0; i < b.size(); i += 32) up.push_back(*std::max_element(b.begin() + i, b.begin() + i + 32));
        while (up.size() % 32) up.push_back(INT32_MIN);
        L.a.push_back(up);
    }
    L.P.ends = L.a[0].data();
    L.P.H = (int)L.a.size() - 1;
    for (int h = 0; h < kMaxLevels; ++h) L.P.m[h] = h < L.P.H ? L.a[h + 1].data() : nullptr;
    return L;
}
int main(int argc, char** argv) {
    const int own = atoi(argv[1]), listed = atoi(argv[2]), cap = 2048;
    std::vector<int32_t> ends(5000), lends(listed), remap(listed);
    for (size_t i = 0; i < ends.size(); ++i) ends[i] = (int32_t)((i * 7919) % 1000);
    for (int i = 0; i < listed; ++i) { lends[i] = (i * 104729) % 1000; remap[i] = 3 * i; }
    const Level A = pyramid(ends), B = pyramid(lends);
    const int64_t lo = 1000, umax = lo + own - 1;
    const int32_t L = 500;
    std::vector<int32_t> pos, end;
    for (int64_t k = umax; k >= lo; --k) if (ends[k] >= L) { pos.push_back((int32_t)k); end.push_back(ends[k]); }
    const int want1 = (int)pos.size();
    for (int k = listed - 1; k >= 0; --k) if (lends[k] >= L) { pos.push_back(remap[k]); end.push_back(lends[k]); }
    const int want2 = (int)pos.size() - want1;
    for (int w = 0; w < kWarpsPerCta; ++w) warp_bar.push_back(std::make_unique<std::barrier<>>(32));
    std::vector<int32_t> cpos(cap + 64), cend(cap + 64), lst(cap + 64), cnt(cap + 64);
    std::vector<uint32_t> msk(cap + 64);
    int s_wsum[kWarpsPerCta], s_n = 0, s_sum = 0, bad = 0;
    std::vector<std::thread> ts;
    std::mutex mu;
    for (int t = 0; t < kThreads; ++t)
        ts.emplace_back([&, t] {
            threadIdx.x = t;
            const int n1 = gather_bfs<int32_t>(A.P, lo, umax, L, cap, cpos.data(), cend.data(), lst.data(), cnt.data(),
                                               msk.data(), s_wsum, &s_n, &s_sum);
            const int n2 = gather_bfs<int32_t>(B.P, 0, listed - 1, L, cap - n1, cpos.data() + n1, cend.data() + n1,
                                               lst.data() + n1, cnt.data(), msk.data(), s_wsum, &s_n, &s_sum,
                                               remap.data());
            std::lock_guard<std::mutex> g(mu);
            if (n1 != want1 || n2 != want2) ++bad;
        });
    for (auto& t : ts) t.join();
    for (size_t i = 0; i < pos.size(); ++i) if (cpos[i] != pos[i] || cend[i] != end[i]) ++bad;
    printf("%d threads or candidates differ\n", bad);
    return bad != 0;
}
"""


def device_function(name, source="si_batched.cu"):
    """The text of a __device__ function, its template line included."""
    text = open(os.path.join(CSRC, source)).read()
    m = re.search(r"^(template <[^\n]*>\n)?__device__ [^\n]*\b%s\(.*?^\}\n" % name, text, re.S | re.M)
    assert m, name
    return m.group(0)


@pytest.fixture(scope="module")
def emulation(tmp_path_factory):
    d = tmp_path_factory.mktemp("gather")
    src, exe = d / "gather.cpp", d / "gather"
    src.write_text(SHIM + device_function("block_excl_scan") + device_function("gather_bfs") + MAIN)
    r = subprocess.run(["g++", "-O1", "-std=c++20", "-pthread", str(src), "-o", str(exe)], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr[:3000]
    return str(exe)


@pytest.mark.parametrize("own,listed", [(0, 40), (1, 1), (20, 20), (20, 900), (31, 2500), (32, 900), (900, 900)])
def test_two_gathers_in_a_row(emulation, own, listed):
    try:
        r = subprocess.run([emulation, str(own), str(listed)], capture_output=True, text=True, timeout=60)
    except subprocess.TimeoutExpired:
        pytest.fail("the block's warps part ways between the two gathers")
    assert r.returncode == 0, r.stdout + r.stderr
