// si_rank.cu -- operations answered from ranks alone, one query per thread in the batch's order:
// counts (count, src/superintervals.hpp:651-825), upper bounds (upper_bound, hpp:501-516) and
// coverage (hpp:979-1006), and the rank grid they read (si_rank.cuh).
#include <algorithm>

#include "si_rank.cuh"

namespace sig {
namespace {

constexpr int kThreads = 256;

// largest g with base[g] <= i
__device__ __forceinline__ int owner(const uint32_t* __restrict__ base, int G, uint32_t i) {
    int lo = 0, hi = G - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (base[mid] <= i) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// buckets a contig of n entries may have (two at least, so that any span fits with a shift below
// 64); its words in t1 are one more
__host__ __device__ __forceinline__ uint32_t grid_cap(int64_t n) {
    const int64_t c = n / kGridFill;
    return (uint32_t)(c > 2 ? c : 2);
}

template <typename S>
__global__ void k_grid_params(const S* __restrict__ arr, const int64_t* __restrict__ seg, int G,
                              const uint32_t* __restrict__ base, GridContig* __restrict__ out) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const int64_t lo = seg[g], hi = seg[g + 1];
    GridContig c{};
    c.lo = (uint32_t)lo;
    c.hi = (uint32_t)hi;
    c.base = base[g];
    if (hi > lo) {
        c.k0 = (int64_t)arr[lo];
        const uint64_t span = (uint64_t)(int64_t)arr[hi - 1] - (uint64_t)c.k0;
        const uint32_t cap = grid_cap(hi - lo);
        uint32_t sh = 0;
        while ((span >> sh) >= cap) ++sh;  // at most 63: span >> 63 is below cap
        c.shift = sh;
        c.nb = (uint32_t)(span >> sh) + 1u;
    }
    out[g] = c;
}

// First position in [a, b) with arr >= v, as offset keys (key - k0, unsigned).
template <typename S>
__device__ __forceinline__ uint32_t first_off(const S* __restrict__ arr, uint32_t a, uint32_t b, int64_t k0,
                                              uint64_t off) {
    uint32_t len = b - a;
    while (len > 0) {
        const uint32_t half = len >> 1;
        const bool below = (uint64_t)(int64_t)arr[a + half] - (uint64_t)k0 < off;
        a = below ? a + half + 1 : a;
        len = below ? len - half - 1 : half;
    }
    return a;
}

// t1: one thread per bucket word, a halving search each.  Neighbouring threads search for
// neighbouring keys, so their reads fall on the same lines.
template <typename S>
__global__ void __launch_bounds__(kThreads) k_grid_fill(const S* __restrict__ arr, int G,
                                                        const uint32_t* __restrict__ base,
                                                        const GridContig* __restrict__ cs, uint32_t words,
                                                        uint32_t* __restrict__ t1) {
    const uint32_t i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= words) return;
    const GridContig c = cs[owner(base, G, i)];
    const uint32_t j = i - c.base;
    if (j > c.nb) return;
    t1[i] = j == 0 ? c.lo : j == c.nb ? c.hi : first_off(arr, c.lo, c.hi, c.k0, (uint64_t)j << c.shift);
}

// t2: one thread per position.  A position of a crowded bucket writes itself to the words of the
// sub-buckets after its predecessor's up to its own (at most 1024), the bucket's last position also
// the rest.  Coalesced reads and no search: 20 M clustered 64-bit keys took 7.6 ms with a warp per
// bucket searching every word.
template <typename S>
__global__ void __launch_bounds__(kThreads) k_grid_sub(const S* __restrict__ arr, const int64_t* __restrict__ seg,
                                                       int G, int64_t n, const GridContig* __restrict__ cs,
                                                       const uint32_t* __restrict__ t1, uint32_t* __restrict__ t2) {
    const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    int g = 0;
    for (int hi = G - 1; g < hi;) {  // largest g with seg[g] <= i
        const int mid = (g + hi + 1) >> 1;
        if (seg[mid] <= i) g = mid;
        else hi = mid - 1;
    }
    const GridContig c = cs[g];
    const uint64_t d = (uint64_t)(int64_t)arr[i] - (uint64_t)c.k0;
    const uint32_t* t = t1 + c.base + (uint32_t)(d >> c.shift);
    const uint32_t a = t[0], e = t[1], cnt = e - a;
    if (cnt < kGridDense) return;
    const int k = grid_sub_bits(cnt, c.shift), ss = (int)c.shift - k;
    const uint32_t nsub = 1u << k, last = nsub - 1u;
    const uint32_t r = (uint32_t)(d >> ss) & last;
    uint32_t from = 0;
    if ((uint32_t)i > a) {
        const uint64_t dp = (uint64_t)(int64_t)arr[i - 1] - (uint64_t)c.k0;
        from = ((uint32_t)(dp >> ss) & last) + 1u;
    }
    uint32_t* __restrict__ w = t2 + grid_sub_base(a);
    for (uint32_t j = from; j <= r; ++j) w[j] = (uint32_t)i;
    if ((uint32_t)i == e - 1u)
        for (uint32_t j = r + 1u; j <= nsub; ++j) w[j] = e;
}

// The positions of one query with start > end that hit, by one warp: the reference's walk 32
// positions at a time (from a miss it goes on at the smallest branch of the chunk's misses).
template <typename S>
__device__ uint32_t warp_walk_count(const MapView<S>& m, int64_t lo, int64_t top, S s, int lane) {
    uint32_t cnt = 0;
    int64_t i = top;
    while (i >= lo) {
        const int64_t k = i - lane;
        const bool valid = k >= lo;
        S e = 0;
        int32_t br = 0;
        if (valid) {
            e = m.ends[k];
            br = m.branch[k];
        }
        const bool hit = valid && s <= e;
        cnt += (uint32_t)__popc(__ballot_sync(kFull, hit));
        const int b = __reduce_min_sync(kFull, valid && !hit ? br : INT32_MAX);
        i = (int64_t)b < i - 32 ? (int64_t)b : i - 32;
    }
    return cnt;
}

// Counts: no interval has start > end, so an interval that ends before qs starts before qe, and
// count = #(start <= qe) - #(end < qs) for every query with qs <= qe.  The others (qs > qe) are
// walked by their warp.
// Bound by random sector reads (ncu at 12.5 M x 12.5 M int32: L2 75%, DRAM 63% of peak, 5.0 TB/s;
// issue 23%).  One query per thread keeps 92% of the warps resident to cover the four dependent
// reads.  12.5 M random queries: 372 us; 990 us through the sorted batch (sort, gather and
// scattered count write).  2-4 or 8-16 entries a bucket instead of 4-8: 408 and 409 us.
template <typename S>
__global__ void __launch_bounds__(kThreads) k_rank_count(MapView<S> m, RankGrid<S> gs, RankGrid<S> ge,
                                                         const S* __restrict__ qs, const S* __restrict__ qe,
                                                         const int32_t* __restrict__ qc, int64_t nq,
                                                         uint32_t* __restrict__ counts, int* d_err) {
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const int lane = threadIdx.x & 31;
    bool walk = false;
    uint32_t cnt = 0, lo = 0, top = 0;
    S s = 0;
    if (q < nq) {
        const int g = qc ? qc[q] : 0;
        if (g < 0 || g >= m.G) {
            atomicCAS(d_err, kDevOk, kDevBadContig);
        } else {
            s = qs[q];
            const S e = qe[q];
            const GridContig c1 = load_contig(gs.c + g), c2 = load_contig(ge.c + g);
            if (s <= e) {
                uint32_t r1, r2;
                grid_two_ranks(gs, c1, e, ge, c2, s, r1, r2);
                cnt = r1 > r2 ? r1 - r2 : 0u;
            } else {
                lo = c1.lo;
                top = grid_first_gt<S>(gs, c1, e);
                walk = top > lo;
            }
        }
    }
    unsigned todo = __ballot_sync(kFull, walk);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const uint32_t r = warp_walk_count<S>(m, (int64_t)__shfl_sync(kFull, lo, src),
                                              (int64_t)__shfl_sync(kFull, top, src) - 1, __shfl_sync(kFull, s, src),
                                              lane);
        if (lane == src) cnt = r;
    }
    if (q < nq) counts[q] = cnt;
}

// 20 M random 64-bit queries over 20 M keys, 70% of both in hotspots: 267 us; 2.31 ms through the
// sorted batch, whose search windows a hotspot overflows.
template <typename S>
__global__ void __launch_bounds__(kThreads) k_rank_ub(RankGrid<S> gs, int G, const S* __restrict__ qe,
                                                      const int32_t* __restrict__ qc, int64_t nq,
                                                      int32_t* __restrict__ out, int* d_err) {
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= nq) return;
    const int g = qc ? qc[q] : 0;
    if (g < 0 || g >= G) {
        atomicCAS(d_err, kDevOk, kDevBadContig);
        out[q] = -1;
        return;
    }
    const GridContig c = load_contig(gs.c + g);
    out[q] = (int32_t)(grid_first_gt<S>(gs, c, qe[q]) - c.lo) - 1;
}

// Coverage of a query with qs <= qe, over the hits {start <= qe} minus {end < qs}:
//   count = a_u - r_qs
//   sum min(end, qe) = PE[r_qe] - PE[r_qs] + qe * (a_u - r_qe)
//   sum max(start, qs) = PS[a_u] - PS[ls] + qs * (ls - r_qs)
// with a_u the first start > qe, r_qs / r_qe the first sorted ends >= qs / > qe, ls the first
// start >= qs, and PS / PE the exclusive prefix sums (mod 2^64) of the starts and of the sorted
// ends.  The coverage, sum min - sum max, wraps as the coordinate type does.
// 5 M x 5 M: 374 us for the call; 853 us through the sorted batch and three block searches.
template <typename S>
__global__ void __launch_bounds__(kThreads) k_rank_cov(RankGrid<S> gs, RankGrid<S> ge, int G,
                                                       const S* __restrict__ qs, const S* __restrict__ qe,
                                                       const int32_t* __restrict__ qc, int64_t nq,
                                                       const uint64_t* __restrict__ ps_start,
                                                       const uint64_t* __restrict__ ps_end,
                                                       uint64_t* __restrict__ count, S* __restrict__ cov, int* d_err,
                                                       int* d_inv) {
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (q >= nq) return;
    const S s = qs[q], e = qe[q];
    if (s > e) *d_inv = 1;
    const int g = qc ? qc[q] : 0;
    if (g < 0 || g >= G || s > e) {
        if (g < 0 || g >= G) atomicCAS(d_err, kDevOk, kDevBadContig);
        count[q] = 0;
        cov[q] = 0;
        return;
    }
    const GridContig c1 = load_contig(gs.c + g), c2 = load_contig(ge.c + g);
    uint32_t a_u, r_qs, r_qe, ls;
    grid_two_ranks(gs, c1, e, ge, c2, s, a_u, r_qs);
    grid_two_ranks(ge, c2, e, gs, c1, s, r_qe, ls);
    const uint64_t qe64 = (uint64_t)(int64_t)e, qs64 = (uint64_t)(int64_t)s;
    const uint64_t smin = ps_end[r_qe] - ps_end[r_qs] + qe64 * ((uint64_t)a_u - (uint64_t)r_qe);
    const uint64_t smax = ps_start[a_u] - ps_start[ls] + qs64 * ((uint64_t)ls - (uint64_t)r_qs);
    count[q] = (uint64_t)a_u - (uint64_t)r_qs;
    cov[q] = (S)(smin - smax);
}

inline unsigned blocks_for(int64_t n) { return (unsigned)std::max<int64_t>(1, ceil_div(n, kThreads)); }

}  // namespace

int64_t grid_t1_words(const int64_t* seg, int G, uint32_t* base) {
    int64_t w = 0;
    for (int g = 0; g < G; ++g) {
        base[g] = (uint32_t)w;
        w += (int64_t)grid_cap(seg[g + 1] - seg[g]) + 1;
    }
    return w;
}

template <typename S>
cudaError_t launch_grid_build(const S* arr, int64_t n, const int64_t* seg, int G, const uint32_t* d_base,
                              int64_t t1_words, GridContig* c, uint32_t* t1, uint32_t* t2, cudaStream_t st) {
    k_grid_params<S><<<blocks_for(G), kThreads, 0, st>>>(arr, seg, G, d_base, c);
    k_grid_fill<S><<<blocks_for(t1_words), kThreads, 0, st>>>(arr, G, d_base, c, (uint32_t)t1_words, t1);
    k_grid_sub<S><<<blocks_for(n), kThreads, 0, st>>>(arr, seg, G, n, c, t1, t2);
    note_launch(3);
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_rank_count(MapView<S> m, RankGrid<S> gs, RankGrid<S> ge, QueryBatch q, uint32_t* counts,
                              int* d_err, cudaStream_t st) {
    if (q.nq <= 0) return cudaSuccess;
    k_rank_count<S><<<blocks_for(q.nq), kThreads, 0, st>>>(m, gs, ge, static_cast<const S*>(q.qs),
                                                           static_cast<const S*>(q.qe), q.qc, q.nq, counts, d_err);
    note_launch();
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_rank_ub(RankGrid<S> gs, int G, const void* qe, const int32_t* qc, int64_t nq, int32_t* out,
                           int* d_err, cudaStream_t st) {
    if (nq <= 0) return cudaSuccess;
    k_rank_ub<S><<<blocks_for(nq), kThreads, 0, st>>>(gs, G, static_cast<const S*>(qe), qc, nq, out, d_err);
    note_launch();
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_rank_coverage(RankGrid<S> gs, RankGrid<S> ge, int G, QueryBatch q, const uint64_t* ps_start,
                                 const uint64_t* ps_end, uint64_t* count, S* cov, int* d_err, int* d_inv,
                                 cudaStream_t st) {
    if (q.nq <= 0) return cudaSuccess;
    k_rank_cov<S><<<blocks_for(q.nq), kThreads, 0, st>>>(gs, ge, G, static_cast<const S*>(q.qs),
                                                         static_cast<const S*>(q.qe), q.qc, q.nq, ps_start, ps_end,
                                                         count, cov, d_err, d_inv);
    note_launch();
    return cudaGetLastError();
}

#define SIG_RINST(S)                                                                                            \
    template cudaError_t launch_grid_build<S>(const S*, int64_t, const int64_t*, int, const uint32_t*, int64_t,  \
                                              GridContig*, uint32_t*, uint32_t*, cudaStream_t);                  \
    template cudaError_t launch_rank_count<S>(MapView<S>, RankGrid<S>, RankGrid<S>, QueryBatch, uint32_t*, int*, \
                                              cudaStream_t);                                                     \
    template cudaError_t launch_rank_ub<S>(RankGrid<S>, int, const void*, const int32_t*, int64_t, int32_t*,     \
                                           int*, cudaStream_t);                                                  \
    template cudaError_t launch_rank_coverage<S>(RankGrid<S>, RankGrid<S>, int, QueryBatch, const uint64_t*,     \
                                                 const uint64_t*, uint64_t*, S*, int*, int*, cudaStream_t);
SIG_RINST(int32_t)
SIG_RINST(int64_t)

}  // namespace sig
