// si_rank.cuh -- rank grid: the rank of a key in each contig's ascending coordinates in one or two
// dependent reads (three to five where coordinates crowd), for queries in any order.
//
// Counts, upper bounds and coverage need only ranks (how many starts / sorted ends lie below a
// key).  A halving search makes log2(n) dependent reads per rank, and sorting the batch first, so
// that neighbours share a search window, costs three radix passes, a gather and a scattered write.
// The grid cuts each contig's coordinate range into power-of-two wide buckets, 4-8 entries each on
// average, with a 16-byte record each: the bucket's first position and, of up to 12 entries, the top
// seven bits of their offsets from the bucket's first coordinate.  A rank is then one 16-byte read and
// a packed compare of the key's own seven bits; only where an entry shares them with the key (1 in 20
// ranks) are those entries compared in full.  Where coordinates crowd, the record of a bucket of more
// entries holds their number; one of kGridDense or more is cut again, by its own count and over its own
// entries' range, in table t2 (by the bucket's range, one outlying coordinate in a 64-bit contig, which
// leaves all others in one bucket, left them in one sub-bucket as well: 12 M counts 1851 us, 467 so).
// Its words sit at 3/8 of the bucket's first position, so that no second index is needed (a bucket of
// n entries uses at most n/4 + 1 words).  Any sub-bucket still crowded is searched by halving: the
// answer is exact for every distribution, only the number of reads changes.
// Full compares take 16-bit offsets inside buckets at most 65536 wide, eight to a 16-byte read, and
// the coordinates elsewhere.  What bounds it is sectors from the L2 (some 9 TB/s of them): the tables
// and offsets of an 8 M-interval index, starts and ends, are some 100 MB, but a rank reads one sector,
// not the two or three of a table of first positions with the offsets beside it.
// Memory: at most 7.5 bytes per entry and array (records 4, t2 1.5, offsets 2), beside 4 or 8 for the
// coordinates.
#pragma once
#include "si_internal.cuh"

namespace sig {

constexpr uint32_t kGridFill = 4;    // at most n / kGridFill buckets: 4-8 entries a bucket
constexpr uint32_t kGridSlots = 12;  // entries whose codes a record holds
constexpr uint32_t kGridMany = 0x80000000u;
constexpr uint32_t kGridOwn = 0x80000000u;
constexpr uint32_t kGridDense = 20;  // entries from which a bucket has its own table (>= 13: see above)

// A contig's buckets.  Its first position is in rec[base], its end in rec[base + nb].
template <typename S>
struct GridContig;
template <>
struct alignas(16) GridContig<int32_t> {
    int32_t k0;      // smallest key
    uint32_t base;   // first record (nb + 1 of them)
    uint32_t nb;     // buckets (0: empty contig)
    uint32_t shift;  // bucket width 2^shift (offsets are kept up to 16)
};
template <>
struct alignas(16) GridContig<int64_t> {
    int64_t k0;
    uint32_t base, nb, shift, pad[3];
};

template <typename S>
struct RankGrid {
    const S* arr = nullptr;          // ascending inside each contig
    const GridContig<S>* c = nullptr;
    // per bucket (then one for the contig's end): x its first position, y to w a byte per entry, unused
    // ones 0xff; of a bucket with more entries x has kGridMany set and y is their number or, with its own
    // table, kGridOwn | log2 of its sub-buckets << 8 | log2 of their width, z and w the offset of its first
    // entry, where they begin
    const uint4* rec = nullptr;
    const uint32_t* t2 = nullptr;
    const uint16_t* lo = nullptr;    // offsets inside buckets of contigs with shift <= 16
};

template <typename S>
__device__ __forceinline__ GridContig<S> load_contig(const GridContig<S>* __restrict__ p) {
    union {
        GridContig<S> c;
        int4 q[sizeof(GridContig<S>) / 16];
    } u;
#pragma unroll
    for (int k = 0; k < (int)(sizeof(GridContig<S>) / 16); ++k) u.q[k] = reinterpret_cast<const int4*>(p)[k];
    return u.c;
}

__device__ __forceinline__ uint32_t grid_sub_base(uint32_t first) { return (uint32_t)((3ull * first + 7) >> 3); }

// Top seven bits of an offset in a bucket 2^shift wide (all of them up to 2^7).
__device__ __forceinline__ uint32_t grid_code(uint64_t d, uint32_t shift) {
    return shift > 7 ? (uint32_t)(d >> (shift - 7)) & 127u : (uint32_t)d & ((1u << shift) - 1u);
}

__device__ __forceinline__ uint32_t grid_first_of(const uint4* __restrict__ rec) {
    return __ldg(reinterpret_cast<const uint32_t*>(rec)) & ~kGridMany;
}

// The record of v's bucket (before the contig: its first one's, behind it: the end's).
template <typename S>
__device__ __forceinline__ uint32_t grid_slot(const GridContig<S>& c, S v) {
    const uint64_t b = ((uint64_t)(int64_t)v - (uint64_t)(int64_t)c.k0) >> c.shift;
    return c.base + (v <= c.k0 ? 0u : b < c.nb ? (uint32_t)b : c.nb);
}

// The positions [a, a + len) among which the first entry >= v of the contig lies (a + len when none
// of them is), x being v's record: len is 0 where the tables alone give the answer.  off: v's offset
// in its bucket.
template <typename S>
__device__ __forceinline__ void grid_bracket(const RankGrid<S>& R, const GridContig<S>& c, S v, uint4 x, uint32_t& a,
                                             uint32_t& len, uint32_t& off) {
    const uint64_t d = (uint64_t)(int64_t)v - (uint64_t)(int64_t)c.k0;
    const bool in = v > c.k0 && (d >> c.shift) < c.nb;
    a = x.x & ~kGridMany;
    len = 0;
    off = (uint32_t)d & ((1u << min(c.shift, 16u)) - 1u);
    if (!in) return;
    if (x.x < kGridMany) {
        // bytes with the top bit set are >= the code (codes have seven bits, so no borrow leaves a
        // byte); taking one more away leaves it where they are above the code
        constexpr uint32_t H = 0x80808080u, one = 0x01010101u;
        const uint32_t q = grid_code(d, c.shift) * one;
        const uint32_t y = (x.y | H) - q, z = (x.z | H) - q, w = (x.w | H) - q;
        const uint32_t lt = (~y & H) | ((~z & H) >> 1) | ((~w & H) >> 2);
        const uint32_t n = (uint32_t)__popc(lt);
        if (c.shift > 7) {
            const uint32_t le = (~(y - one) & ~x.y & H) | ((~(z - one) & ~x.z & H) >> 1) | ((~(w - one) & ~x.w & H) >> 2);
            len = (uint32_t)__popc(le) - n;
        }
        a += n;
        return;
    }
    if (x.y < kGridOwn) {
        len = x.y;
        return;
    }
    const uint64_t in_bucket = d & ((1ull << c.shift) - 1ull), first = (uint64_t)x.w << 32 | x.z;
    if (in_bucket <= first) return;
    const uint64_t r = (in_bucket - first) >> (x.y & 63u);
    const uint32_t nsub = 1u << ((x.y >> 8) & 31u);
    const uint32_t* t2 = R.t2 + grid_sub_base(a) + (r < nsub ? (uint32_t)r : nsub);
    a = __ldg(t2);
    // (behind the last sub-bucket the bucket's end is the answer, and where one is a coordinate wide every
    // entry of v's equals v)
    if (r < nsub && (x.y & 63u) != 0u) len = __ldg(t2 + 1) - a;
}

// Entries of v's bucket among the eight from `at` (a multiple of 8) on that lie in [a, a + len) and
// below v (offset off): one 16-byte read and four packed compares.
__device__ __forceinline__ uint32_t grid_block8(const uint16_t* __restrict__ lo, uint32_t at, uint32_t a, uint32_t len,
                                                uint32_t off2) {
    const uint4 x = __ldg(reinterpret_cast<const uint4*>(lo + at));
    uint32_t below = (__vcmpltu2(x.x, off2) & 0x00010001u) | (__vcmpltu2(x.y, off2) & 0x00020002u) |
                     (__vcmpltu2(x.z, off2) & 0x00040004u) | (__vcmpltu2(x.w, off2) & 0x00080008u);
    // bits 0-3: entries 0, 2, 4, 6; bits 16-19: entries 1, 3, 5, 7
    const int f = (int)(a - at), l = (int)(a + len - at);  // [f, l) of the block counts
    const uint32_t from = f <= 0 ? 0u : (uint32_t)f, to = l >= 8 ? 8u : (uint32_t)l;
    const uint32_t even = ((1u << ((to + 1) >> 1)) - 1u) & ~((1u << ((from + 1) >> 1)) - 1u);
    const uint32_t odd = ((1u << (to >> 1)) - 1u) & ~((1u << (from >> 1)) - 1u);
    below &= even | (odd << 16);
    return (uint32_t)__popc(below);
}

// The first of the positions [a, a + len) of v's bucket whose entry is >= v (a + len when none).
template <typename S>
__device__ __forceinline__ uint32_t grid_inside(const RankGrid<S>& R, const GridContig<S>& c, S v, uint32_t a,
                                                uint32_t len, uint32_t off) {
    if (c.shift <= 16) {
        while (len > 8) {
            const uint32_t half = len >> 1;
            const bool below = (uint32_t)__ldg(R.lo + a + half) < off;
            a = below ? a + half + 1 : a;
            len = below ? len - half - 1 : half;
        }
        if (len > 0) {
            const uint32_t at = a & ~7u, off2 = off | (off << 16);
            uint32_t n = grid_block8(R.lo, at, a, len, off2);
            if (a + len > at + 8) n += grid_block8(R.lo, at + 8, a, len, off2);
            a += n;
        }
    } else {
        while (len > 0) {
            const uint32_t half = len >> 1;
            const bool below = __ldg(R.arr + a + half) < v;
            a = below ? a + half + 1 : a;
            len = below ? len - half - 1 : half;
        }
    }
    return a;
}

// First position of the contig with arr >= v (its end when none).
template <typename S>
__device__ __forceinline__ uint32_t grid_first_geq(const RankGrid<S>& R, const GridContig<S>& c, S v) {
    uint32_t a, len, off;
    grid_bracket(R, c, v, __ldg(R.rec + grid_slot(c, v)), a, len, off);
    return grid_inside(R, c, v, a, len, off);
}

// First position with arr > v.
template <typename S>
__device__ __forceinline__ uint32_t grid_first_gt(const RankGrid<S>& R, const GridContig<S>& c, S v) {
    return v == Lim<S>::hi ? grid_first_of(R.rec + c.base + c.nb) : grid_first_geq<S>(R, c, (S)(v + 1));
}

// The key whose first_geq is v's first_gt, where there is one.
template <typename S>
__device__ __forceinline__ S grid_after(S v) {
    return v == Lim<S>::hi ? v : (S)(v + 1);
}

// first_gt(v1) in one array and first_geq(v2) in another, x1 and x2 being the records of
// grid_after(v1) and v2.
template <typename S>
__device__ __forceinline__ void grid_two_ranks(const RankGrid<S>& R1, const GridContig<S>& c1, S v1, uint4 x1,
                                               const RankGrid<S>& R2, const GridContig<S>& c2, S v2, uint4 x2,
                                               uint32_t& r1, uint32_t& r2) {
    uint32_t a1, l1, o1, a2, l2, o2;
    const S w1 = grid_after(v1);
    grid_bracket(R1, c1, w1, x1, a1, l1, o1);
    grid_bracket(R2, c2, v2, x2, a2, l2, o2);
    r1 = grid_inside(R1, c1, w1, a1, l1, o1);
    r2 = grid_inside(R2, c2, v2, a2, l2, o2);
    if (v1 == Lim<S>::hi) r1 = grid_first_of(R1.rec + c1.base + c1.nb);
}

// Records for contigs of these sizes (fills base[g]), and words of t2 for n entries.
int64_t grid_records(const int64_t* seg, int G, uint32_t* base);
inline int64_t grid_t2_words(int64_t n) { return (3 * n + 7) / 8 + 8; }
// Builds the tables over arr (ascending inside each contig): d_base holds grid_records' bases.
template <typename S>
cudaError_t launch_grid_build(const S* arr, int64_t n, const int64_t* seg, int G, const uint32_t* d_base,
                              int64_t records, GridContig<S>* c, uint4* rec, uint32_t* t2, uint16_t* lo,
                              cudaStream_t st);

// Counts of a batch in its own order, for an index without intervals with start > end.
template <typename S>
cudaError_t launch_rank_count(MapView<S> m, RankGrid<S> gs, RankGrid<S> ge, QueryBatch q, uint32_t* counts,
                              int* d_err, cudaStream_t st);
// Counts and their exclusive prefix sums (off, n + 1 entries) in one pass, and each query's upper
// bound (su: the first position whose start exceeds the query's end, 0 when no start of its contig
// is at or below it or the contig is outside [0, G)).  work: rank_work_bytes(nq), zeroed by the call
// unless it is `cleared`.
// With pieces, a query with start > end counts nothing (it gives no piece of an intersection).
struct RankWork {
    int err;                   // device error word
    int inv;                   // free for the caller
    unsigned long long total;  // hits of the batch
    unsigned int longest;      // hits of its query with the most
    unsigned int tiles;        // tile counter
    unsigned int walked;       // progress of the walks of queries with start > end
    unsigned int pad[9];
};
size_t rank_work_bytes(int64_t nq);
template <typename S>
cudaError_t launch_rank_scan(MapView<S> m, RankGrid<S> gs, RankGrid<S> ge, QueryBatch q, bool pieces, uint32_t* su,
                             int64_t* off, RankWork* work, cudaStream_t st, bool cleared = false);
// The direct emit's lanes per query for a batch of nq queries and P hits, `longest` of them of one query,
// over n intervals, 0 for the sorted tiles; below far_below hits most of them are long intervals lying
// far apart (see direct_lanes).  A query's walk is a chain of dependent reads: some 400 ns a chunk of
// `lanes` positions, 600 ns a far hit, however many other queries there are.  The tiles, which write
// such a query's hits by stretches, take 77 us, 190 ps a query, 20 ps an interval and 11 ps a hit in all; the
// direct emit is left to batches whose longest walk ends sooner (1 M queries over 5 M intervals with
// 3 hits each: 0.2 ms, and 54 ms when one of them had 400 k).
__host__ __device__ inline int rank_lanes(int64_t n, int64_t far_below, int64_t nq, int64_t P, int64_t longest) {
    const bool far = P < far_below;
    if (far ? P > 4000000 + 10 * nq + n || P > 160 * nq : P > 7000000 + 17 * nq + 9 * n / 5) return 0;
    const int lanes = nq <= (far ? 4096 : P > 30 * nq ? 524288 : 32768) ? 32
                      : nq <= 262144 || (!far && P > 16 * nq)           ? 8
                                                                        : 2;
    const int64_t walk_ps = far ? 600000 * longest : 400000 / lanes * longest;
    return walk_ps > 77000000 + 190 * nq + 20 * n + 11 * P ? 0 : lanes;
}
// An emit queued behind launch_rank_scan before the host knows the hit count: every block reads the
// count and leaves when the batch failed, when the output has no room or when rank_lanes names
// another kernel; the host, which reads the same record after both, then goes that other way.  It
// saves the wait between the two kernels: 100 k searches with 0.7 hits each 60 -> 45 us.
struct EmitGate {
    const RankWork* work = nullptr;    // null: emit
    int64_t room = 0;                  // results that the output holds
    int64_t n = 0, far_below = 0;      // rank_lanes
};
// What the direct emit writes for each hit.
enum RankOut : int { kOutIdx = 0, kOutValue = 1, kOutKeys = 2, kOutPieces = 3 };
template <typename S>
struct RankDest {
    int32_t* i32 = nullptr;  // positions, payloads or (keys: may be null) payloads
    S* s = nullptr;          // keys, pieces: starts
    S* e = nullptr;          // and ends
};
// Writes every query's hits at off[q] - out_base, by groups of `lanes` (2, 8 or 32) lanes per query.
template <typename S>
cudaError_t launch_rank_emit(MapView<S> m, QueryBatch q, const uint32_t* su, const int64_t* off, int64_t out_base,
                             int order, int what, RankDest<S> d, int lanes, int* d_err, cudaStream_t st,
                             EmitGate gate = EmitGate());

// Gaps: the stretches of each contig's coordinate range that no interval covers (no interval has
// start > end).  Slots: contig g's positions, then one after its last; flags mark those with a gap
// before them, offs are the flags' exclusive prefix sums.
template <typename S>
cudaError_t launch_gap_flags(MapView<S> m, uint32_t* flags, cudaStream_t st);
cudaError_t launch_gap_seg(const int64_t* offs, const int64_t* seg, int G, int64_t* gap_seg, cudaStream_t st);
template <typename S>
cudaError_t launch_gap_write(MapView<S> m, const uint32_t* flags, const int64_t* offs, S* gs, S* ge, cudaStream_t st);
// The gaps that each query meets, clipped to it: the off[q + 1] - off[q] gaps before su[q].
template <typename S>
cudaError_t launch_gap_emit(const S* gs, const S* ge, QueryBatch q, const uint32_t* su, const int64_t* off, S* os,
                            S* oe, cudaStream_t st, EmitGate gate = EmitGate());

// Contig-local upper bounds (-1: none) of every query end.
template <typename S>
cudaError_t launch_rank_ub(RankGrid<S> gs, int G, const void* qe, const int32_t* qc, int64_t nq, int32_t* out,
                           int* d_err, cudaStream_t st);
// Coverage from ranks and prefix sums (see launch site); *d_inv is set when a query has start > end
// (it is answered 0 and 0, and the caller computes the batch another way).
template <typename S>
cudaError_t launch_rank_coverage(RankGrid<S> gs, RankGrid<S> ge, int G, QueryBatch q, const uint64_t* ps_start,
                                 const uint64_t* ps_end, uint64_t* count, S* cov, int* d_err, int* d_inv,
                                 cudaStream_t st);

}  // namespace sig
