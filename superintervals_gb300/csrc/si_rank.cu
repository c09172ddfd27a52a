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
// 64); its records are one more
__host__ __device__ __forceinline__ uint32_t grid_cap(int64_t n) {
    const int64_t c = n / kGridFill;
    return (uint32_t)(c > 2 ? c : 2);
}

constexpr int kSamples = 64;

template <typename S>
__global__ void k_grid_params(const S* __restrict__ arr, const int64_t* __restrict__ seg, int G,
                              const uint32_t* __restrict__ base, GridContig<S>* __restrict__ out) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= G) return;
    const int64_t lo = seg[g], hi = seg[g + 1];
    GridContig<S> c{};
    c.base = base[g];
    if (hi > lo) {
        c.k0 = arr[lo];
        const uint64_t span = (uint64_t)(int64_t)arr[hi - 1] - (uint64_t)(int64_t)arr[lo];
        // records for the entries outside the crowded stretches: the others, at least four times as
        // dense as the whole, get sub-tables, and a smaller table stays closer (gaps of 5 M intervals,
        // 5 M differences: 270 us with a record per four gaps throughout, 257 so)
        int spread = 0;
        S from = c.k0;
#pragma unroll 8
        for (int k = 1; k <= kSamples; ++k) {
            const S to = arr[lo + (hi - lo - 1) * k / kSamples];
            spread += (uint64_t)(int64_t)to - (uint64_t)(int64_t)from >= span / (4 * kSamples) ? 1 : 0;
            from = to;
        }
        const uint32_t cap = grid_cap((hi - lo) * spread / kSamples);
        uint32_t sh = 0;
        while ((span >> sh) >= cap) ++sh;  // at most 63: span >> 63 is below cap
        c.shift = sh;
        c.nb = (uint32_t)(span >> sh) + 1u;
    }
    out[g] = c;
}

// First position in [a, b) with arr >= k0 + off.
template <typename S>
__device__ __forceinline__ uint32_t first_off(const S* __restrict__ arr, uint32_t a, uint32_t b, S k0, uint64_t off) {
    uint32_t len = b - a;
    while (len > 0) {
        const uint32_t half = len >> 1;
        const bool below = (uint64_t)(int64_t)arr[a + half] - (uint64_t)(int64_t)k0 < off;
        a = below ? a + half + 1 : a;
        len = below ? len - half - 1 : half;
    }
    return a;
}

// Records: one thread each, a halving search for the bucket's first position (neighbouring threads
// search for neighbouring keys, so their reads fall on the same lines), then its entries' codes.  A
// block's last thread only finds the end of the one before.
template <typename S>
__global__ void __launch_bounds__(kThreads) k_grid_fill(const S* __restrict__ arr, const int64_t* __restrict__ seg,
                                                        int G, const uint32_t* __restrict__ base,
                                                        const GridContig<S>* __restrict__ cs, uint32_t records,
                                                        uint4* __restrict__ rec) {
    __shared__ uint32_t s_at[kThreads];
    const uint32_t i = blockIdx.x * (kThreads - 1) + threadIdx.x;
    uint32_t at = 0, j = 0;
    GridContig<S> c{};
    if (i < records) {
        const int g = owner(base, G, i);
        c = cs[g];
        j = i - c.base;
        const uint32_t lo = (uint32_t)seg[g], hi = (uint32_t)seg[g + 1];
        at = j == 0 ? lo : j >= c.nb ? hi : first_off(arr, lo, hi, c.k0, (uint64_t)j << c.shift);
    }
    s_at[threadIdx.x] = at;
    __syncthreads();
    if (threadIdx.x == kThreads - 1 || i >= records || j > c.nb) return;
    const uint32_t cnt = j < c.nb ? s_at[threadIdx.x + 1] - at : 0u;
    uint4 x = make_uint4(at, ~0u, ~0u, ~0u);
    if (cnt >= kGridDense) {
        // as many sub-buckets as a quarter of the entries, or fewer, over the entries' own range
        const uint64_t in_bucket = (1ull << c.shift) - 1ull;
        const uint64_t first = ((uint64_t)(int64_t)arr[at] - (uint64_t)(int64_t)c.k0) & in_bucket;
        const uint64_t last = ((uint64_t)(int64_t)arr[at + cnt - 1] - (uint64_t)(int64_t)c.k0) & in_bucket;
        const uint32_t bits = 31 - __clz(cnt >> 2);
        uint32_t ss = 0;
        while (((last - first) >> ss) >> bits) ++ss;
        x = make_uint4(at | kGridMany, kGridOwn | bits << 8 | ss, (uint32_t)first, (uint32_t)(first >> 32));
    } else if (cnt > kGridSlots) {
        x = make_uint4(at | kGridMany, cnt, 0u, 0u);
    } else {
        uint32_t w[3] = {~0u, ~0u, ~0u};
#pragma unroll
        for (uint32_t k = 0; k < kGridSlots; ++k)
            if (k < cnt) {
                const uint32_t code = grid_code((uint64_t)(int64_t)arr[at + k] - (uint64_t)(int64_t)c.k0, c.shift);
                w[k >> 2] ^= (code ^ 0xffu) << (8 * (k & 3));
            }
        x = make_uint4(at, w[0], w[1], w[2]);
    }
    rec[i] = x;
}

// Offsets and t2: one thread per position.  A position of a bucket with its own table writes itself to
// the words of the sub-buckets after its predecessor's up to its own, the bucket's last position also
// the rest; stretches of more than kOwnWords words (a gap in a large bucket) are written by the block.
// Coalesced reads and no search: 20 M clustered 64-bit keys took 7.6 ms with a warp per bucket
// searching every word.
constexpr uint32_t kOwnWords = 64;
template <typename S>
__global__ void __launch_bounds__(kThreads) k_grid_sub(const S* __restrict__ arr, const int64_t* __restrict__ seg,
                                                       int G, int64_t n, const GridContig<S>* __restrict__ cs,
                                                       const uint4* __restrict__ rec, uint32_t* __restrict__ t2,
                                                       uint16_t* __restrict__ lo) {
    __shared__ uint32_t s_from[2 * kThreads], s_len[2 * kThreads], s_val[2 * kThreads];
    __shared__ unsigned int s_n;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    auto fill = [&](uint32_t at, uint32_t len, uint32_t val) {
        if (len <= kOwnWords) {
            for (uint32_t j = 0; j < len; ++j) t2[at + j] = val;
        } else {
            const unsigned int k = atomicAdd(&s_n, 1u);  // a thread has two stretches at most
            s_from[k] = at;
            s_len[k] = len;
            s_val[k] = val;
        }
    };
    if (i < n) {
        int g = 0;
        for (int hi = G - 1; g < hi;) {  // largest g with seg[g] <= i
            const int mid = (g + hi + 1) >> 1;
            if (seg[mid] <= i) g = mid;
            else hi = mid - 1;
        }
        const GridContig<S> c = cs[g];
        const uint64_t d = (uint64_t)(int64_t)arr[i] - (uint64_t)(int64_t)c.k0;
        lo[i] = (uint16_t)((uint32_t)d & ((1u << min(c.shift, 16u)) - 1u));
        const uint32_t at = c.base + (uint32_t)(d >> c.shift);
        const uint4 x = rec[at];
        if (x.x >= kGridMany && x.y >= kGridOwn) {
            const uint32_t a = x.x & ~kGridMany, e = rec[at + 1].x & ~kGridMany;  // the bucket [a, e)
            const uint32_t ss = x.y & 63u, nsub = 1u << ((x.y >> 8) & 31u);
            const uint64_t in_bucket = (1ull << c.shift) - 1ull, first = (uint64_t)x.w << 32 | x.z;
            const uint32_t r = (uint32_t)(((d & in_bucket) - first) >> ss);
            uint32_t from = 0;
            if ((uint32_t)i > a) {
                const uint64_t dp = (uint64_t)(int64_t)arr[i - 1] - (uint64_t)(int64_t)c.k0;
                from = (uint32_t)(((dp & in_bucket) - first) >> ss) + 1u;
            }
            const uint32_t w = grid_sub_base(a);
            if (from <= r) fill(w + from, r + 1u - from, (uint32_t)i);
            if ((uint32_t)i == e - 1u) fill(w + r + 1u, nsub - r, e);
        }
    }
    __syncthreads();
    for (unsigned int k = 0; k < s_n; ++k)
        for (uint32_t j = threadIdx.x; j < s_len[k]; j += kThreads) t2[s_from[k] + j] = s_val[k];
}

// The positions of a warp's queries with start > end (walk) that hit, from top - 1 down to lo.  Several
// at once: each lane walks its own a little way, which ends most of them (a warp's 32 one after another:
// 1000 such queries over 1 M intervals 104 us, 26 so).  What is left the warp walks together, one query
// after the other: the reference's walk 32 positions at a time (from a miss it goes on at the smallest
// branch of the chunk's misses).  A walk is as long as its hits are many; it counts every kBeatChunks
// chunks in *walked (null: nobody waits for the warp).  A function of its own: inlined, the rare walks
// cost the scan kernel up to eight registers a thread.
constexpr int kOwnSteps = 64;
constexpr uint32_t kBeatChunks = 256;
template <typename S>
__device__ __noinline__ uint32_t warp_walks(const S* __restrict__ ends, const int32_t* __restrict__ branch, uint32_t lo,
                                            uint32_t top, S s, bool walk, unsigned int* walked) {
    const int lane = threadIdx.x & 31;
    uint32_t cnt = 0;
    unsigned todo = __ballot_sync(kFull, walk);
    if (__popc(todo) > 2) {
        int64_t i = (int64_t)top - 1;
        for (int k = 0; k < kOwnSteps && walk; ++k) {
            const bool hit = s <= ends[i];
            const int32_t br = branch[i];
            cnt += hit ? 1u : 0u;
            i = hit ? i - 1 : (int64_t)br;
            walk = i >= (int64_t)lo;
        }
        top = (uint32_t)(i + 1);
        todo = __ballot_sync(kFull, walk);
    }
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const int64_t last = __shfl_sync(kFull, lo, src);
        const S key = __shfl_sync(kFull, s, src);
        uint32_t r = 0, chunks = 0;
        for (int64_t i = (int64_t)__shfl_sync(kFull, top, src) - 1; i >= last;) {
            if (++chunks % kBeatChunks == 0 && walked && lane == 0) atomicAdd(walked, 1u);
            const int64_t k = i - lane;
            const bool valid = k >= last;
            S e = 0;
            int32_t br = 0;
            if (valid) {
                e = ends[k];
                br = branch[k];
            }
            const bool hit = valid && key <= e;
            r += (uint32_t)__popc(__ballot_sync(kFull, hit));
            const int b = __reduce_min_sync(kFull, valid && !hit ? br : INT32_MAX);
            i = (int64_t)b < i - 32 ? (int64_t)b : i - 32;
        }
        if (lane == src) cnt += r;
    }
    return cnt;
}

// One query and the records of its two ranks (g < 0: none, or a contig outside the index).
template <typename S>
struct RankQuery {
    int g = -1;
    S s = 0, e = 0;
    uint4 x1, x2;
};
template <typename S>
__device__ __forceinline__ void rank_load(const MapView<S>& m, const S* __restrict__ qs, const S* __restrict__ qe,
                                          const int32_t* __restrict__ qc, int64_t q, int64_t nq, int* d_err,
                                          RankQuery<S>& Q) {
    if (q >= nq) return;
    const int g = qc ? qc[q] : 0;
    Q.s = qs[q];
    Q.e = qe[q];
    if (g >= 0 && g < m.G) Q.g = g;
    else atomicCAS(d_err, kDevOk, kDevBadContig);
}
template <typename S>
__device__ __forceinline__ void rank_probe(const RankGrid<S>& gs, const RankGrid<S>& ge, RankQuery<S>& Q) {
    const int g = max(Q.g, 0);
    Q.x1 = __ldg(gs.rec + grid_slot(load_contig(gs.c + g), grid_after(Q.e)));
    Q.x2 = __ldg(ge.rec + grid_slot(load_contig(ge.c + g), Q.s));
}

// The query's count (see k_rank_count) and upper bound; the warp's queries with start > end are
// walked by the whole warp, so every lane of the warp calls it (walked: see warp_walks).
template <typename S>
__device__ __forceinline__ uint32_t rank_one(const MapView<S>& m, const RankGrid<S>& gs, const RankGrid<S>& ge,
                                             const RankQuery<S>& Q, bool pieces, uint32_t& upper,
                                             unsigned int* walked) {
    bool walk = false;
    uint32_t cnt = 0, lo = 0, top = 0;
    const S s = Q.s, e = Q.e;
    upper = 0;
    if (Q.g >= 0) {
        const GridContig<S> c1 = load_contig(gs.c + Q.g);
        const bool any = c1.nb != 0 && e >= c1.k0;  // some start at or below the query's end
        if (s <= e) {
            uint32_t r2;
            grid_two_ranks(gs, c1, e, Q.x1, ge, load_contig(ge.c + Q.g), s, Q.x2, top, r2);
            cnt = top > r2 ? top - r2 : 0u;
        } else {
            top = grid_first_gt<S>(gs, c1, e);
            walk = !pieces && any;
            lo = walk ? (uint32_t)m.seg[Q.g] : 0u;
        }
        upper = any && (s <= e || !pieces) ? top : 0u;
    }
    if (__any_sync(kFull, walk)) cnt += warp_walks<S>(m.ends, m.branch, lo, top, s, walk, walked);
    return cnt;
}

// Counts: no interval has start > end, so an interval that ends before qs starts before qe, and
// count = #(start <= qe) - #(end < qs) for every query with qs <= qe.  The others (qs > qe) are
// walked by their warp.
// Bound by random sector reads (ncu at 12.5 M x 12.5 M int32: 5 L2 sectors a query, two of them the
// records, which come from DRAM for the larger part: 1.08 GB, 61% of its peak; issue 46%).  One query
// per thread keeps 84% of the warps resident.  12.5 M random queries: 205 us, with both records read
// before either is used (226 else); 990 us through the sorted batch (sort, gather and scattered count
// write).  With first positions in one table and the offsets in another 267 us (halving over the
// coordinates instead: 371), with a record per 3 or 6 entries 3% less and 13% more.  Contig records
// in shared memory cost 20 us.
template <typename S>
__global__ void __launch_bounds__(kThreads) k_rank_count(MapView<S> m, RankGrid<S> gs, RankGrid<S> ge,
                                                         const S* __restrict__ qs, const S* __restrict__ qe,
                                                         const int32_t* __restrict__ qc, int64_t nq,
                                                         uint32_t* __restrict__ counts, int* d_err) {
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    uint32_t upper;
    RankQuery<S> Q;
    rank_load(m, qs, qe, qc, q, nq, d_err, Q);
    rank_probe(gs, ge, Q);
    const uint32_t cnt = rank_one<S>(m, gs, ge, Q, false, upper, nullptr);
    if (q < nq) counts[q] = cnt;
}

// 20 M random 64-bit queries over 20 M keys, 70% of both in hotspots: 241 us (218 with a table of first
// positions, whose words are four times as close in the hotspots); 2.31 ms through the
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
    const GridContig<S> c = load_contig(gs.c + g);
    const uint32_t r = grid_first_gt<S>(gs, c, qe[q]);
    out[q] = (int32_t)(r - (qc ? grid_first_of(gs.rec + c.base) : 0u)) - 1;  // without contig ids: contig 0
}

// Coverage of a query with qs <= qe, over the hits {start <= qe} minus {end < qs}:
//   count = a_u - r_qs
//   sum min(end, qe) = PE[r_qe] - PE[r_qs] + qe * (a_u - r_qe)
//   sum max(start, qs) = PS[a_u] - PS[ls] + qs * (ls - r_qs)
// with a_u the first start > qe, r_qs / r_qe the first sorted ends >= qs / > qe, ls the first
// start >= qs, and PS / PE the exclusive prefix sums (mod 2^64) of the starts and of the sorted
// ends.  The coverage, sum min - sum max, wraps as the coordinate type does.
// 5 M x 5 M: 225 us for the call; 853 us through the sorted batch and three block searches.
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
    const GridContig<S> c1 = load_contig(gs.c + g), c2 = load_contig(ge.c + g);
    uint32_t a_u, r_qs, r_qe, ls;
    const S after = grid_after(e);
    grid_two_ranks(gs, c1, e, __ldg(gs.rec + grid_slot(c1, after)), ge, c2, s, __ldg(ge.rec + grid_slot(c2, s)), a_u,
                   r_qs);
    grid_two_ranks(ge, c2, e, __ldg(ge.rec + grid_slot(c2, after)), gs, c1, s, __ldg(gs.rec + grid_slot(c1, s)), r_qe,
                   ls);
    const uint64_t qe64 = (uint64_t)(int64_t)e, qs64 = (uint64_t)(int64_t)s;
    const uint64_t smin = ps_end[r_qe] - ps_end[r_qs] + qe64 * ((uint64_t)a_u - (uint64_t)r_qe);
    const uint64_t smax = ps_start[a_u] - ps_start[ls] + qs64 * ((uint64_t)ls - (uint64_t)r_qs);
    count[q] = (uint64_t)a_u - (uint64_t)r_qs;
    cov[q] = (S)(smin - smax);
}

// Look-back status of a tile: 2 flag bits over a 62-bit sum.
constexpr unsigned long long kTileAgg = 1ull << 62;  // the tile's own total
constexpr unsigned long long kTilePre = 2ull << 62;  // the total of this and all earlier tiles
constexpr unsigned long long kTileVal = (1ull << 62) - 1ull;
constexpr int kSpinLimit = 1 << 22;                  // polls of one window without progress before giving up

__device__ __forceinline__ void st_tile(unsigned long long* p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_tile(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned int ld_word(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Counts and offsets in one pass: a block takes the next tile of kThreads * R queries from an atomic
// counter, counts them, publishes the tile's total, and its first warp looks back over the earlier
// tiles' published totals, 32 at a time, until an inclusive prefix (decoupled look-back).  A tile of
// queries with start > end publishes only when it has walked their hits (1024 queries of 4 M hits
// each: seconds), so a window that stays unpublished for kSpinLimit polls is given up, with
// kDevTimeout, only when no walk of the launch went on meanwhile; a walk ends at its contig's first
// position, so the kernel always ends.  Against the count kernel and a scan it saves a launch, a
// cleared buffer and the counts' way through memory.  (The bounds on the registers, 32, 40 and 48, are what
// the kernel takes without the call to the walks.)
template <typename S, int R>
__global__ void __launch_bounds__(kThreads, R == 1 ? 8 : sizeof(S) == 4 ? 6 : 5) k_rank_scan(MapView<S> m, RankGrid<S> gs, RankGrid<S> ge,
                                                        const S* __restrict__ qs, const S* __restrict__ qe,
                                                        const int32_t* __restrict__ qc, int64_t nq, int pieces,
                                                        uint32_t* __restrict__ su, int64_t* __restrict__ off,
                                                        RankWork* __restrict__ work) {
    constexpr int kWarps = kThreads / kWarp;
    __shared__ int64_t s_warp[kWarps];
    __shared__ unsigned int s_most[kWarps];
    __shared__ int64_t s_prefix;
    __shared__ unsigned int s_t;
    unsigned long long* status = reinterpret_cast<unsigned long long*>(work + 1);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_t = atomicAdd(&work->tiles, 1u);  // tiles in start order: earlier tiles run
    __syncthreads();
    const int64_t t = s_t;
    const int64_t base = t * (kThreads * R) + (int64_t)w * (R * kWarp) + lane;
    int64_t v[R];
    int64_t carry = 0;
    unsigned int most = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t q = base + r * kWarp;
        uint32_t upper;
        RankQuery<S> Q;
        rank_load(m, qs, qe, qc, q, nq, &work->err, Q);
        rank_probe(gs, ge, Q);
        const int64_t x = rank_one<S>(m, gs, ge, Q, pieces != 0, upper, &work->walked);
        if (q < nq) su[q] = upper;
        most = max(most, __reduce_max_sync(kFull, (unsigned int)x));
        int64_t inc = x;
#pragma unroll
        for (int d = 1; d < kWarp; d <<= 1) {
            const int64_t y = __shfl_up_sync(kFull, inc, d);
            if (lane >= d) inc += y;
        }
        v[r] = carry + inc - x;
        carry += __shfl_sync(kFull, inc, 31);
    }
    if (lane == 0) {
        s_warp[w] = carry;
        s_most[w] = most;
    }
    __syncthreads();
    if (w == 0) {
        int64_t total = 0;
#pragma unroll
        for (int k = 0; k < kWarps; ++k) {
            total += s_warp[k];
            most = max(most, s_most[k]);
        }
        if (lane == 0) st_tile(status + t, (t == 0 ? kTilePre : kTileAgg) | (unsigned long long)total);
        int64_t excl = 0;
        if (t > 0) {
            int64_t top = t - 1;
            int spins = 0;
            unsigned int walked = 0;
            while (true) {
                const int64_t p = top - lane;
                const unsigned long long s = p >= 0 ? ld_tile(status + p) : kTilePre;
                const unsigned long long f = s & ~kTileVal;
                if (__any_sync(kFull, f == 0ull)) {
                    if (++spins > kSpinLimit) {
                        const unsigned int now = __shfl_sync(kFull, ld_word(&work->walked), 0);
                        if (now == walked) {
                            if (lane == 0) atomicCAS(&work->err, kDevOk, kDevTimeout);
                            break;
                        }
                        walked = now;
                        spins = 0;
                    }
                    __nanosleep(32);
                    continue;
                }
                spins = 0;
                const unsigned pm = __ballot_sync(kFull, f == kTilePre);
                const int first = pm ? __ffs(pm) - 1 : 32;
                int64_t x = lane <= first ? (int64_t)(s & kTileVal) : 0;
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) x += __shfl_xor_sync(kFull, x, d);
                excl += x;
                if (pm) break;
                top -= 32;
            }
            if (lane == 0) st_tile(status + t, kTilePre | (unsigned long long)(excl + total));
        }
        if (lane == 0) {
            s_prefix = excl;
            if ((t + 1) * (kThreads * R) >= nq) {  // the last tile
                off[nq] = excl + total;
                work->total = (unsigned long long)(excl + total);
            }
            atomicMax(&work->longest, most);  // nobody waits for it
        }
    }
    __syncthreads();
    int64_t o = s_prefix;
    for (int k = 0; k < w; ++k) o += s_warp[k];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t q = base + r * kWarp;
        if (q < nq) off[q] = v[r] + o;
    }
}

// Direct emit: the hits of each query written by W lanes in the batch's own order, from its known
// upper bound and count.  The lanes look at W positions at a time, downwards; the walk ends with the
// last hit (the count says which), and goes on below a chunk at the smallest branch of its misses
// (from a miss at p every position above branch[p] ends before ends[p] < qs).  Neighbouring
// queries' lists are neighbours in the output, so the writes coalesce across the warp's groups.
// Right for sparse results: a tile of queries far apart shares nothing, and sorting the batch
// costs more than the hits.  Bound by the dependent reads of the walk (about 12-16 ps a hit with the
// device full; lanes per query: see direct_lanes).  Whole calls, before (sorted tiles) and after:
// 100 k queries with 0.7 hits each 205 -> 45 us, 3 M with 2.7 hits 1290 -> 289 us, 3 M with 33 hits
// 1418 -> 1130 us; 3 M with 126 hits would go 2306 -> 5551 us.
template <typename S, int W, int OUT>
__global__ void __launch_bounds__(kThreads) k_rank_emit(MapView<S> m, const S* __restrict__ qs,
                                                        const S* __restrict__ qe, const int32_t* __restrict__ qc,
                                                        int64_t nq, const uint32_t* __restrict__ su,
                                                        const int64_t* __restrict__ off, int64_t out_base, int order,
                                                        RankDest<S> dst, int* d_err, EmitGate gate) {
    __shared__ int s_open;
    if (gate.work) {  // by one thread, not by every warp
        if (threadIdx.x == 0) {
            const int64_t P = (int64_t)gate.work->total;
            s_open = !gate.work->err && P <= gate.room &&
                     rank_lanes(gate.n, gate.far_below, nq, P, gate.work->longest) == W;
        }
        __syncthreads();
        if (!s_open) return;
    }
    const int lane = threadIdx.x & 31, sub = lane & (W - 1);
    const unsigned gmask = W == 32 ? kFull : ((1u << (W & 31)) - 1u) << (lane & ~(W - 1));
    const int64_t q = ((int64_t)blockIdx.x * kThreads + threadIdx.x) / W;
    int64_t at = 0;
    int cnt = 0, i = -1, lo = 0;
    S s = 0, e0 = 0;
    if (q < nq) {
        at = off[q];
        cnt = (int)(off[q + 1] - at);
        at -= out_base;
        if (cnt > 0) {
            i = (int)su[q] - 1;
            s = qs[q];
            if (OUT == kOutPieces) e0 = qe[q];
            const int g = qc ? qc[q] : 0;
            lo = (int)m.seg[g];
        }
    }
    const bool ascending = order == kOrderIdxsCpp;
    int done = 0;      // hits written
    int head = -1;     // length of the head run (ascending order only)
    while (true) {
        const bool active = done < cnt && i >= lo;  // group-uniform
        if (!__any_sync(kFull, active)) break;
        const int k = i - sub;
        const bool in = active && k >= lo;
        S e = 0;
        if (in) e = m.ends[k];
        const bool hit = in && s <= e;
        const unsigned bal = __ballot_sync(kFull, hit);
        const unsigned mine = (bal & gmask) >> (lane & ~(W - 1));
        if (ascending && __any_sync(kFull, active && head < 0)) {
            // the head run: consecutive hits from the upper bound down; it goes on below this chunk
            // only when the whole chunk hits
            const unsigned full = W == 32 ? kFull : (1u << (W & 31)) - 1u;
            bool open = active && head < 0;
            int h = mine == full ? W : __ffs(~mine) - 1;
            bool more = open && mine == full && h < cnt;
            while (__any_sync(kFull, more)) {
                const int k2 = i - h - sub;
                const bool hit2 = more && k2 >= lo && s <= m.ends[k2];
                const unsigned b2 = (__ballot_sync(kFull, hit2) & gmask) >> (lane & ~(W - 1));
                if (more) {
                    h += b2 == full ? W : __ffs(~b2) - 1;
                    more = b2 == full && h < cnt;
                }
            }
            if (open) head = h;
        }
        const int rank = done + __popc(mine & ((1u << sub) - 1u));
        if (hit && rank < cnt) {
            const int64_t p = at + (rank < head ? head - 1 - rank : rank);
            if constexpr (OUT == kOutIdx) {
                dst.i32[p] = k - lo;
            } else if constexpr (OUT == kOutValue) {
                dst.i32[p] = m.data[k];
            } else if constexpr (OUT == kOutKeys) {
                dst.s[p] = m.starts[k];
                dst.e[p] = e;
                if (dst.i32) dst.i32[p] = m.data[k];
            } else {
                const S st = m.starts[k];
                dst.s[p] = st > s ? st : s;
                dst.e[p] = e < e0 ? e : e0;
                dst.i32[p] = k - lo;
            }
        }
        done += __popc(mine);
        // the next chunk, where hits are left
        int next = i - W;
        if (__any_sync(kFull, active && done < cnt)) {
            int br = INT32_MAX;
            if (in && !hit && done < cnt) br = m.branch[k];
#pragma unroll
            for (int d = W / 2; d > 0; d >>= 1) br = min(br, __shfl_xor_sync(kFull, br, d));
            next = min(next, br);
        }
        if (active) i = next;
    }
    if (done != cnt && sub == 0) atomicCAS(d_err, kDevOk, kDevOverflow);  // internal: count and walk differ
}

// ---- gaps (difference, hpp:1186-1211) -------------------------------------------------------
// All intervals before position i end before start[i] - 1 exactly when the i smallest ends of the
// contig do (an interval from i on ends at or after start[i]), i.e. when end_sorted[i - 1] does: a
// gap lies before i when end_sorted[i - 1] + 1 < start[i], and it is [end_sorted[i - 1] + 1,
// start[i] - 1].  One elementwise pass over two arrays finds the complement of the union.
template <typename S>
__device__ __forceinline__ bool gap_before(const MapView<S>& m, int64_t slot, S& a, S& b) {
    int g = 0;
    for (int hi = m.G - 1; g < hi;) {  // largest g with its first slot seg[g] + g <= slot
        const int mid = (g + hi + 1) >> 1;
        if (m.seg[mid] + mid <= slot) g = mid;
        else hi = mid - 1;
    }
    const int64_t lo = m.seg[g], hi = m.seg[g + 1], i = slot - g;
    a = Lim<S>::lo;
    b = Lim<S>::hi;
    if (i > lo) {
        const S e = m.end_sorted[i - 1];
        if (e == Lim<S>::hi) return false;
        a = (S)(e + 1);
    }
    if (i < hi) {
        const S s = m.starts[i];
        if (s == Lim<S>::lo) return false;
        b = (S)(s - 1);
    }
    return a <= b;
}

template <typename S>
__global__ void __launch_bounds__(kThreads) k_gap_flags(MapView<S> m, int64_t slots, uint32_t* __restrict__ flags) {
    const int64_t t = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= slots) return;
    S a, b;
    flags[t] = gap_before(m, t, a, b) ? 1u : 0u;
}

__global__ void k_gap_seg(const int64_t* __restrict__ offs, const int64_t* __restrict__ seg, int G,
                          int64_t* __restrict__ out) {
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g <= G) out[g] = offs[seg[g] + g];
}

template <typename S>
__global__ void __launch_bounds__(kThreads) k_gap_write(MapView<S> m, int64_t slots,
                                                        const uint32_t* __restrict__ flags,
                                                        const int64_t* __restrict__ offs, S* __restrict__ gs,
                                                        S* __restrict__ ge) {
    const int64_t t = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= slots || !flags[t]) return;
    S a, b;
    gap_before(m, t, a, b);
    gs[offs[t]] = a;
    ge[offs[t]] = b;
}

// One warp writes the pieces of 32 neighbouring queries, which lie one after another in the output:
// lane l takes every 32nd piece of the warp's stretch and finds its query among the 32 by halving
// over their offsets (shuffles), so writes coalesce and a query of many pieces is shared by all lanes.
// gridDim.y warps share a stretch, 32 pieces in turn, where the batch has fewer stretches than the device
// warps: 300 queries with 20 k pieces each are ten stretches, 4.2 ms by a warp each, the call 116 us by 64.
// 5 M queries against 5 M intervals: the whole call 1856 us with hit lists swept per query, 257 us
// from the gaps.
template <typename S>
__global__ void __launch_bounds__(kThreads) k_gap_emit(const S* __restrict__ gs, const S* __restrict__ ge,
                                                       const S* __restrict__ qs, const S* __restrict__ qe, int64_t nq,
                                                       const uint32_t* __restrict__ su,
                                                       const int64_t* __restrict__ off, S* __restrict__ os,
                                                       S* __restrict__ oe, EmitGate gate) {
    if (gate.work && (gate.work->err || (int64_t)gate.work->total > gate.room)) return;
    const int lane = threadIdx.x & 31;
    const int64_t q = (int64_t)blockIdx.x * kThreads + threadIdx.x;
    const bool live = q < nq;
    const int64_t mine = live ? off[q] : off[nq];
    const int64_t next = live ? off[q + 1] : mine;
    const int64_t first = __shfl_sync(kFull, mine, 0), last = __shfl_sync(kFull, next, 31);
    // lanes past the batch hold empty queries at its end
    uint32_t top = 0;
    S s = 0, e = 0;
    if (next > mine) {
        top = su[q];
        s = qs[q];
        e = qe[q];
    }
    for (int64_t p0 = first + 32 * (int64_t)blockIdx.y; p0 < last; p0 += 32 * (int64_t)gridDim.y) {
        const int64_t p = p0 + lane;
        int k = 0;  // the last query of the warp whose offset is <= p
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const int64_t o = __shfl_sync(kFull, mine, k + d);
            if (o <= p) k += d;
        }
        const uint32_t t = __shfl_sync(kFull, top, k);
        const int64_t end = __shfl_sync(kFull, next, k);
        const S s0 = __shfl_sync(kFull, s, k), e0 = __shfl_sync(kFull, e, k);
        if (p < last) {
            const uint32_t at = t - (uint32_t)(end - p);
            const S a = gs[at], b = ge[at];
            os[p] = a > s0 ? a : s0;
            oe[p] = b < e0 ? b : e0;
        }
    }
}

inline unsigned blocks_for(int64_t n) { return (unsigned)std::max<int64_t>(1, ceil_div(n, kThreads)); }

}  // namespace

int64_t grid_records(const int64_t* seg, int G, uint32_t* base) {
    int64_t w = 0;
    for (int g = 0; g < G; ++g) {
        base[g] = (uint32_t)w;
        w += (int64_t)grid_cap(seg[g + 1] - seg[g]) + 1;
    }
    return w;
}

template <typename S>
cudaError_t launch_grid_build(const S* arr, int64_t n, const int64_t* seg, int G, const uint32_t* d_base,
                              int64_t records, GridContig<S>* c, uint4* rec, uint32_t* t2, uint16_t* lo,
                              cudaStream_t st) {
    k_grid_params<S><<<blocks_for(G), kThreads, 0, st>>>(arr, seg, G, d_base, c);
    k_grid_fill<S><<<(unsigned)ceil_div(records, (int64_t)kThreads - 1), kThreads, 0, st>>>(arr, seg, G, d_base, c,
                                                                                           (uint32_t)records, rec);
    k_grid_sub<S><<<blocks_for(n), kThreads, 0, st>>>(arr, seg, G, n, c, rec, t2, lo);
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

// queries per tile of the count and scan kernel: one per thread while the batch fits the device
// about once, else four, for fewer look-backs
constexpr int64_t kScanSmall = 152 * 2048;

size_t rank_work_bytes(int64_t nq) {
    const int64_t tiles = ceil_div(nq > 0 ? nq : 1, nq <= kScanSmall ? kThreads : 4 * kThreads);
    return sizeof(RankWork) + sizeof(unsigned long long) * (size_t)tiles;
}

template <typename S>
cudaError_t launch_rank_scan(MapView<S> m, RankGrid<S> gs, RankGrid<S> ge, QueryBatch q, bool pieces, uint32_t* su,
                             int64_t* off, RankWork* work, cudaStream_t st, bool cleared) {
    if (!cleared) {
        cudaError_t e = cudaMemsetAsync(work, 0, rank_work_bytes(q.nq), st);
        if (e != cudaSuccess) return e;
    }
    if (q.nq <= 0) return cudaMemsetAsync(off, 0, sizeof(int64_t), st);
    const S* qs = static_cast<const S*>(q.qs);
    const S* qe = static_cast<const S*>(q.qe);
    if (q.nq <= kScanSmall)
        k_rank_scan<S, 1><<<blocks_for(q.nq), kThreads, 0, st>>>(m, gs, ge, qs, qe, q.qc, q.nq, pieces, su, off, work);
    else
        k_rank_scan<S, 4><<<(unsigned)ceil_div(q.nq, 4 * kThreads), kThreads, 0, st>>>(m, gs, ge, qs, qe, q.qc, q.nq,
                                                                                      pieces, su, off, work);
    note_launch();
    return cudaGetLastError();
}

template <typename S, int W>
static cudaError_t rank_emit_w(MapView<S> m, QueryBatch q, const uint32_t* su, const int64_t* off, int64_t out_base,
                               int order, int what, RankDest<S> d, int* d_err, cudaStream_t st, EmitGate gate) {
    const unsigned blocks = blocks_for(q.nq * W);
    const S* qs = static_cast<const S*>(q.qs);
    const S* qe = static_cast<const S*>(q.qe);
    switch (what) {
        case kOutIdx:
            k_rank_emit<S, W, kOutIdx><<<blocks, kThreads, 0, st>>>(m, qs, qe, q.qc, q.nq, su, off, out_base, order, d, d_err, gate);
            break;
        case kOutValue:
            k_rank_emit<S, W, kOutValue><<<blocks, kThreads, 0, st>>>(m, qs, qe, q.qc, q.nq, su, off, out_base, order, d, d_err, gate);
            break;
        case kOutKeys:
            k_rank_emit<S, W, kOutKeys><<<blocks, kThreads, 0, st>>>(m, qs, qe, q.qc, q.nq, su, off, out_base, order, d, d_err, gate);
            break;
        default:
            k_rank_emit<S, W, kOutPieces><<<blocks, kThreads, 0, st>>>(m, qs, qe, q.qc, q.nq, su, off, out_base, order, d, d_err, gate);
    }
    note_launch();
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_rank_emit(MapView<S> m, QueryBatch q, const uint32_t* su, const int64_t* off, int64_t out_base,
                             int order, int what, RankDest<S> d, int lanes, int* d_err, cudaStream_t st,
                             EmitGate gate) {
    if (q.nq <= 0) return cudaSuccess;
    if (lanes == 2) return rank_emit_w<S, 2>(m, q, su, off, out_base, order, what, d, d_err, st, gate);
    if (lanes == 8) return rank_emit_w<S, 8>(m, q, su, off, out_base, order, what, d, d_err, st, gate);
    return rank_emit_w<S, 32>(m, q, su, off, out_base, order, what, d, d_err, st, gate);
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

template <typename S>
cudaError_t launch_gap_flags(MapView<S> m, uint32_t* flags, cudaStream_t st) {
    k_gap_flags<S><<<blocks_for(m.n + m.G), kThreads, 0, st>>>(m, m.n + m.G, flags);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_gap_seg(const int64_t* offs, const int64_t* seg, int G, int64_t* gap_seg, cudaStream_t st) {
    k_gap_seg<<<blocks_for(G + 1), kThreads, 0, st>>>(offs, seg, G, gap_seg);
    note_launch();
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_gap_write(MapView<S> m, const uint32_t* flags, const int64_t* offs, S* gs, S* ge,
                             cudaStream_t st) {
    k_gap_write<S><<<blocks_for(m.n + m.G), kThreads, 0, st>>>(m, m.n + m.G, flags, offs, gs, ge);
    note_launch();
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_gap_emit(const S* gs, const S* ge, QueryBatch q, const uint32_t* su, const int64_t* off, S* os,
                            S* oe, cudaStream_t st, EmitGate gate) {
    if (q.nq <= 0) return cudaSuccess;
    const int64_t split = 152 * 32 / ceil_div(q.nq, kWarp);  // of 32 warps on each SM
    const dim3 grid(blocks_for(q.nq), (unsigned)std::min<int64_t>(std::max<int64_t>(split, 1), 64));
    k_gap_emit<S><<<grid, kThreads, 0, st>>>(gs, ge, static_cast<const S*>(q.qs), static_cast<const S*>(q.qe), q.nq,
                                             su, off, os, oe, gate);
    note_launch();
    return cudaGetLastError();
}

#define SIG_RINST(S)                                                                                            \
    template cudaError_t launch_grid_build<S>(const S*, int64_t, const int64_t*, int, const uint32_t*, int64_t,  \
                                              GridContig<S>*, uint4*, uint32_t*, uint16_t*, cudaStream_t);          \
    template cudaError_t launch_rank_count<S>(MapView<S>, RankGrid<S>, RankGrid<S>, QueryBatch, uint32_t*, int*, \
                                              cudaStream_t);                                                     \
    template cudaError_t launch_rank_scan<S>(MapView<S>, RankGrid<S>, RankGrid<S>, QueryBatch, bool, uint32_t*,  \
                                             int64_t*, RankWork*, cudaStream_t, bool);                           \
    template cudaError_t launch_rank_emit<S>(MapView<S>, QueryBatch, const uint32_t*, const int64_t*, int64_t,   \
                                             int, int, RankDest<S>, int, int*, cudaStream_t, EmitGate);          \
    template cudaError_t launch_rank_ub<S>(RankGrid<S>, int, const void*, const int32_t*, int64_t, int32_t*,     \
                                           int*, cudaStream_t);                                                  \
    template cudaError_t launch_rank_coverage<S>(RankGrid<S>, RankGrid<S>, int, QueryBatch, const uint64_t*,     \
                                                 const uint64_t*, uint64_t*, S*, int*, int*, cudaStream_t);
#define SIG_GINST(S)                                                                                           \
    template cudaError_t launch_gap_flags<S>(MapView<S>, uint32_t*, cudaStream_t);                            \
    template cudaError_t launch_gap_write<S>(MapView<S>, const uint32_t*, const int64_t*, S*, S*, cudaStream_t); \
    template cudaError_t launch_gap_emit<S>(const S*, const S*, QueryBatch, const uint32_t*, const int64_t*, S*, \
                                            S*, cudaStream_t, EmitGate);
SIG_GINST(int32_t)
SIG_GINST(int64_t)
SIG_RINST(int32_t)
SIG_RINST(int64_t)

}  // namespace sig
