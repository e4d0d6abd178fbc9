// Order-free exact accumulation for PlusTimes<double> SpGEMM columns.
//
// The reference folds each output entry as acc = add(mrhs, acc) over the B
// column's entries in ascending order (mtSpGEMM.h:396-412).  In fp64 that
// left fold is order dependent, so reproducing it on the GPU forces every
// product of one row to be applied in k order.  These kernels remove the
// order instead: every product p = fl(a * b) (rounded exactly as the
// reference rounds it) is an integer multiple of 2^(ebase - 1075), where
// ebase is the smallest product exponent of the column, so the column's
// products are added EXACTLY as integers, and each output entry is the exact
// sum rounded once to the nearest double (ties to even).  Integer addition
// is associative, so any interleaving of the products -- lane-parallel
// shared-memory atomics from all warps, unsorted buckets -- gives the same
// bits: repeated runs are bit-identical, and each value is the correctly
// rounded sum of the reference's own products, within the reference's own
// summation error of its hash-path and heap-path results.
//
// Accumulator: one signed 128-bit integer per output row, in four 32-bit words
// of shared memory (word i the multiples of 2^(32 i)); a product's 53-bit
// mantissa covers at most three words, added with 32-bit shared atomics whose
// returned old value says whether a carry (a borrow, for a negative product)
// goes on to the next word.  A column is admitted when all its products are
// normal and finite and
//   span <= kXOMax                       (every product has its words)
//   span + 53 + lg(nnz(B(:,j))) <= 125   (the exact sum fits 126 bits)
// with span = (largest - smallest product exponent) bounded from per-column
// exponent ranges of A and the B values; other columns (subnormal values,
// possible underflow, inf/nan, very wide ranges) are listed for the ordered
// kernel.
#pragma once

#include <stdint.h>

#include <type_traits>

#include "semiring.cuh"
#include "spgemm_kernels.cuh"

namespace gbc {

constexpr int kXOMax = 61;       // largest product exponent above the base
constexpr int kXRows = 4096;     // rows of a row tile, and output rows of one accumulator pass
constexpr int kXThreads = 512;   // two blocks per SM

// Per column of A: smallest and largest biased exponent of its nonzero
// values, each plus kXBias in 12 bits, kXMixed when a value is negative or
// zero, and kXZero when one is zero.  Subnormal values count as exponent -64 (their products can
// underflow: such columns take the ordered kernel); a column without nonzero
// values gets min > max.
constexpr int kXBias = 64;
constexpr uint32_t kXMixed = 1u << 24;
constexpr uint32_t kXZero = 1u << 25;

static __global__ void k_aexp_f64(int64_t ncol, const int64_t *acp, const double *aval, int32_t *aexp)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t c = warp; c < ncol; c += nwarps) {
        int lo = 4095 - kXBias, hi = -kXBias;
        bool mixed = false, zeros = false;
        for (int64_t p = acp[c] + lane; p < acp[c + 1]; p += 32) {
            const uint64_t bits = (uint64_t)__double_as_longlong(aval ? aval[p] : 1.0);
            int e = (int)((bits >> 52) & 0x7ff);
            const bool zero = (bits << 1) == 0;
            mixed |= zero || (bits >> 63);
            zeros |= zero;
            if (e == 0) e = -kXBias;
            if (!zero) {
                lo = min(lo, e);
                hi = max(hi, e);
            }
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        mixed = __any_sync(0xffffffffu, mixed);
        zeros = __any_sync(0xffffffffu, zeros);
        if (lane == 0)
            aexp[c] = (int32_t)((uint32_t)(lo + kXBias) | ((uint32_t)(hi + kXBias) << 12) | (mixed ? kXMixed : 0u) |
                                (zeros ? kXZero : 0u));
    }
}

// Add the nonzero product with bit pattern `bits` (normal, of an admitted
// column) to the 128-bit integer whose word i is acc[i * stride].  Words that
// overflow pass their carry on, so no word is ever normalised: the integer is
// exact modulo 2^128 once every thread has finished.  POS: the product is
// positive.  Returns false when the product lies outside the column's
// exponent window (cannot happen for admitted columns; nothing is added then).
template <bool POS>
__device__ __forceinline__ bool x_add128(uint32_t *acc, int stride, uint64_t bits, int ebase)
{
    const uint32_t ml = (uint32_t)bits, h = (uint32_t)(bits >> 32);
    const uint32_t mh = (h & 0xFFFFFu) | 0x100000u;
    const uint32_t o = (POS ? h >> 20 : (h >> 20) & 0x7ffu) - (uint32_t)ebase;
    if (o > (uint32_t)kXOMax) return false;
    const uint32_t p0 = ml << (o & 31);
    const uint32_t p1 = __funnelshift_l(ml, mh, o);
    const uint32_t p2 = __funnelshift_l(mh, 0u, o);  // below 2^21
    uint32_t *w = acc + (o >> 5) * stride;
    if (POS || !(h >> 31)) {
        uint32_t old = atomicAdd(w, p0), t1, wrap, t2, c;
        // t1 = p1 + carry (wrap: p1 was all ones and the carry goes on)
        asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, 0, 0;\n\t}"
            : "=r"(t1), "=r"(wrap)
            : "r"(old), "r"(p0), "r"(p1));
        old = atomicAdd(w + stride, t1);
        asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %1, %2;\n\taddc.u32 %0, %3, %4;\n\t}"
            : "=r"(t2)
            : "r"(old), "r"(t1), "r"(p2), "r"(wrap));
        if (t2) {
            old = atomicAdd(w + 2 * stride, t2);
            c = old > ~t2;
            if (c && o < 32) atomicAdd(w + 3 * stride, 1u);
        }
    } else {
        uint32_t old = atomicAdd(w, 0u - p0);
        uint32_t c = old < p0;
        const uint32_t t1 = p1 + c, wrap = t1 < c;
        old = atomicAdd(w + stride, 0u - t1);
        c = wrap | (uint32_t)(old < t1);
        const uint32_t t2 = p2 + c;
        if (t2) {
            old = atomicAdd(w + 2 * stride, 0u - t2);
            if (old < t2 && o < 32) atomicAdd(w + 3 * stride, ~0u);
        }
    }
    return true;
}

// Round a signed 128-bit integer M (two's complement hi:lo), times
// 2^(ebase - 1075), to the nearest double (ties to even), in integer
// arithmetic (IEEE 754 rounding of the exact value; GB300's fp64 units are
// slow).  flag bit 1 says whether some term was other than -0.0: an exact
// zero sum is then +0.0, else -0.0 (what the left fold of the reference
// gives).  For admitted columns |M| < 2^126 and the result is finite.
__device__ __forceinline__ double x_round(uint64_t hi, uint64_t lo, uint32_t flag, int ebase)
{
    const bool neg = (int64_t)hi < 0;
    if (neg) {
        lo = ~lo + 1;
        hi = ~hi + (lo == 0 ? 1ull : 0ull);
    }
    if ((hi | lo) == 0) return (flag & 2) ? 0.0 : -0.0;
    const int n = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo);  // zeros above |M|'s top bit
    const int e = 127 - n + ebase - 52;  // biased exponent when the result is normal
    uint64_t bits;
    if (e <= 0) {
        // subnormal: |M| * 2^(ebase - 1) < 2^52 is the exact subnormal mantissa
        bits = lo << (ebase - 1);
    } else {
        // |M| shifted to bit 127: 53 bits kept, 11 in `rem`, the others in `rest`
        const uint64_t top = n < 64 ? (hi << n) | ((lo >> 1) >> (63 - n)) : lo << (n - 64);
        const uint64_t rest = n < 64 ? lo << n : 0ull;
        const uint32_t rem = (uint32_t)top & 0x7FFu;
        uint64_t m = top >> 11;
        m += (rem > 0x400u || (rem == 0x400u && (rest != 0 || (m & 1)))) ? 1 : 0;  // 2^53 carries into the exponent
        bits = ((uint64_t)(e - 1) << 52) + m;
    }
    return __longlong_as_double((long long)(bits | (neg ? (1ull << 63) : 0ull)));
}

// Add product p (a double of an admitted column) exactly to a register
// accumulator hi:lo (units of 2^(ebase - 1075)); flag as in x_add.  False
// when p is outside the window.
__device__ __forceinline__ bool x_acc128(uint64_t &hi, uint64_t &lo, uint32_t &flag, double p, int ebase)
{
    const uint64_t bits = (uint64_t)__double_as_longlong(p);
    const int ex = (int)((bits >> 52) & 0x7ff);
    if (bits != (1ull << 63)) flag |= 2;
    if (ex == 0) return (bits << 1) == 0;
    const int o = ex - ebase;
    if ((unsigned)o > (unsigned)kXOMax) return false;
    const uint64_t m = (bits & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const uint64_t pl = m << o;
    const uint64_t ph = o ? (m >> (64 - o)) : 0ull;
    if (bits >> 63) {
        const uint64_t old = lo;
        lo -= pl;
        hi -= ph + (old < pl ? 1ull : 0ull);
    } else {
        lo += pl;
        hi += ph + (lo < pl ? 1ull : 0ull);
    }
    return true;
}

// Exponent window of one B entry's products (A column k's value range
// times b): updates emin (smallest product exponent) and emax (largest,
// allowing for rounding up).  Entries whose products are all zero are skipped.
__device__ __forceinline__ void x_window(int32_t ae, double b, bool has_b, int &emin, int &emax)
{
    const int amin = (int)(ae & 0xfff) - kXBias, amax = (int)((ae >> 12) & 0xfff) - kXBias;
    const uint64_t bb = has_b ? (uint64_t)__double_as_longlong(b) : 0x3FF0000000000000ull;
    int eb = (int)((bb >> 52) & 0x7ff);
    if (amin > amax || (bb << 1) == 0) return;
    if (eb == 0) eb = -64;  // subnormal b
    emin = min(emin, amin + eb - 1023);
    emax = max(emax, amax + eb - 1022);
}

// Is a column with product exponents in [ebase, etop] and nb B entries
// summed exactly?  (Every product normal and finite, every piece inside the
// words, the exact sum inside 126 bits, the rounded result finite.)  An
// all-zero column (ebase > etop) is admitted with ebase 1.
__device__ __forceinline__ bool x_admit(int &ebase, int etop, int64_t nb)
{
    if (ebase > etop) {
        ebase = 1;
        return true;
    }
    const int lg = 64 - __clzll((long long)nb);
    return ebase >= 1 && etop <= 2046 - lg - 2 && (etop - ebase) <= kXOMax && (etop - ebase) + 53 + lg <= 125;
}

// Per column k of A, its row tiles as a compressed list (the DCSC of the
// column's tile structure): entries ptr[k] .. ptr[k+1]-1 hold, for each
// touched tile in order, the tile and the first position of A(:,k) inside
// it, followed by one end marker (tile 0xFFFF, start = the column's end).
static __global__ void k_ktl_count(int64_t ncol, const uint64_t *amask, int mask_words, int64_t *cnt)
{
    const int64_t c = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= ncol) return;
    int64_t n = 1;
    for (int w = 0; w < mask_words; ++w) n += __popcll(amask[c * mask_words + w]);
    cnt[c] = n;
}

// One warp per column; lanes test 32 tiles at a time.
static __global__ void k_ktl_fill(int64_t ncol, const uint32_t *tptr, int T, const int64_t *ptr, uint32_t *kstart,
                           uint16_t *ktile)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t c = warp; c < ncol; c += nwarps) {
        const uint32_t *tp = tptr + c * (int64_t)(T + 1);
        int64_t o = ptr[c];
        for (int t0 = 0; t0 < T; t0 += 32) {
            const int t = t0 + lane;
            const bool nz = t < T && tp[t + 1] > tp[t];
            const unsigned m = __ballot_sync(0xffffffffu, nz);
            if (nz) {
                const int64_t q = o + __popc(m & ((1u << lane) - 1));
                kstart[q] = tp[t];
                ktile[q] = (uint16_t)t;
            }
            o += __popc(m);
        }
        if (lane == 0) {
            kstart[o] = tp[T];
            ktile[o] = 0xFFFF;
        }
    }
}

// One segment of a bucketed column: A's positions [start, start + len)
// (one row tile of one A column) times the column's B entry e.
struct XSeg {
    uint32_t start, len, e;
};

constexpr int kXTMax = 256;                   // row tiles of a bucketed column
constexpr int kXSegs = 1024;                  // segments of one chunk table
constexpr int kXWins = 512;                   // 32-product windows of one round
constexpr int kXSpanTiles = 16;               // row tiles of one ranked visit (a 64 K-row bitmap)
constexpr int kXSort = 4096;                  // products of one sorted range visit (at most)
constexpr int kXLight = 512;                  // runs of at most this many products go to sorted ranges
constexpr int kXDirect = 8192;                // a tile of more products is a visit of its own
constexpr int64_t kXScap = int64_t(1) << 20;  // bucketed segments of one column, at most (per-block scratch)

// Values of up to 8 bytes travel through the chunk tables as bits.
template <typename V>
__device__ __forceinline__ uint64_t x_bits(V v)
{
    uint64_t u = 0;
    memcpy(&u, &v, sizeof(V));
    return u;
}

template <typename V>
__device__ __forceinline__ V x_from(uint64_t u)
{
    V v;
    memcpy(&v, &u, sizeof(V));
    return v;
}

// What k_numeric_x keeps in an output row's accumulator, for the semirings
// whose add does not depend on the order (words 0 when untouched, word i at
// w[i * R]): PlusTimes<double> is x_add128; whole-number sums are two words
// with a carry; minima are the complement of an order-preserving key, so that
// zero is the empty one and a larger key the better; or is a flag.
template <class SR>
struct XAcc {
    static constexpr bool kUse = false;
};

template <>
struct XAcc<PlusTimes<double>> {
    static constexpr bool kUse = true;
};

template <>
struct XAcc<PlusTimes<int64_t>> {
    static constexpr bool kUse = true;
    static __device__ __forceinline__ bool add(uint32_t *w, int R, int at, int64_t p)
    {
        const uint32_t lo = (uint32_t)p, hi = (uint32_t)((uint64_t)p >> 32);
        const uint32_t old = atomicAdd(w + at, lo);
        const uint32_t t = hi + (old > ~lo ? 1u : 0u);
        if (t) atomicAdd(w + R + at, t);
        return true;
    }
    static __device__ __forceinline__ int64_t take(uint32_t *w, int R, int at)
    {
        const uint64_t v = w[at] | ((uint64_t)w[R + at] << 32);
        w[at] = 0;
        w[R + at] = 0;
        return (int64_t)v;
    }
};

template <>
struct XAcc<BoolOrAnd> {
    static constexpr bool kUse = true;
    static __device__ __forceinline__ bool add(uint32_t *w, int, int at, uint8_t p)
    {
        if (p) w[at] = 1;  // every writer writes the same
        return true;
    }
    static __device__ __forceinline__ uint8_t take(uint32_t *w, int, int at)
    {
        const uint8_t v = (uint8_t)w[at];
        w[at] = 0;
        return v;
    }
};

__device__ __forceinline__ void x_max(uint32_t *w, int at, unsigned long long key)
{
    unsigned long long *a = reinterpret_cast<unsigned long long *>(w) + at;
    if (key > *reinterpret_cast<volatile unsigned long long *>(a)) atomicMax(a, key);
}

__device__ __forceinline__ uint64_t x_take(uint32_t *w, int at)
{
    uint64_t *a = reinterpret_cast<uint64_t *>(w) + at;
    const uint64_t k = *a;
    *a = 0;
    return k;
}

struct XMinI64 {
    static constexpr bool kUse = true;
    static __device__ __forceinline__ bool add(uint32_t *w, int, int at, int64_t p)
    {
        x_max(w, at, ~((uint64_t)p ^ (1ull << 63)));
        return true;
    }
    static __device__ __forceinline__ int64_t take(uint32_t *w, int, int at)
    {
        return (int64_t)(~x_take(w, at) ^ (1ull << 63));
    }
};

template <>
struct XAcc<MinPlus<int64_t>> : XMinI64 {};
template <>
struct XAcc<Select2ndMin<int64_t>> : XMinI64 {};

// A NaN or -0.0 among the products makes the fold in order differ from the
// minimum: add() says so, and the column goes to the ordered kernel.
template <>
struct XAcc<MinPlus<double>> {
    static constexpr bool kUse = true;
    static __device__ __forceinline__ bool add(uint32_t *w, int, int at, double p)
    {
        const uint64_t b = (uint64_t)__double_as_longlong(p);
        x_max(w, at, ~(b ^ (b >> 63 ? ~0ull : 1ull << 63)));
        return p == p && b != 1ull << 63;
    }
    static __device__ __forceinline__ double take(uint32_t *w, int, int at)
    {
        const uint64_t k = ~x_take(w, at);
        return __longlong_as_double((long long)(k ^ (k >> 63 ? 1ull << 63 : ~0ull)));
    }
};

// Shared memory of one k_numeric_x block.
struct XSmem {
    uint32_t acc[4 * kXRows];              // accumulator words, plane by plane
    uint32_t bm[kXSpanTiles * kXRows / 32];   // touched rows of the visit
    uint16_t pre[kXSpanTiles * kXRows / 32];  // touched rows before each bitmap word
    uint16_t rows[kXRows];                 // row (from the visit's first) of every accumulator
    uint32_t term[kXRows / 32];            // accumulators with a term other than -0.0 (columns with zeros)
    uint64_t bv[kXSegs];                   // chunk table: bits of the B value of each segment,
    uint32_t base[kXSegs];                 //   segment start - products before it (modulo 2^32),
    int32_t off[kXSegs + 1];               //   products before each segment
    int32_t nseg;                          //   segments
    uint2 win[kXWins];                     // per 32 products: bit i set where a segment starts at the i-th, and
                                           //   the segments that start before the window
    int32_t segcnt[kXTMax], prodcnt[kXTMax], tend[kXTMax];
    int32_t wsum[2][kXThreads / 32];
    int32_t emin[kXThreads / 32], emax[kXThreads / 32], wzero[kXThreads / 32];
    int64_t col;
    int32_t ebase;    // the column's smallest product exponent
    int64_t bs, be;   // its B entries
    int64_t *oir;     // its output
    void *oval;
    int32_t lim;      // output entries it may write
    SpgemmArgs a;
};

// Numeric pass for the columns of the big list, one block per column (dynamic
// counter), for PlusTimes<double> under the exact fold and the semirings whose
// add does not depend on the order (XAcc).  After the column's exponent window
// is admitted (exact sums):
//  1. bucketing -- every (B entry, touched row tile of its A column) pair is
//     counted per tile (segments and products) and written, in any order,
//     into the block's scratch grouped by tile (a counting sort; the exact
//     sum makes the order irrelevant).  Each tile is then visited with its
//     own segments only, instead of looking up every B entry per tile.
//  2. visits in row order, each a chunk table of its segments over which the
//     products are spread evenly:
//      * direct: a tile of more than kXDirect products (or too many segments)
//        is visited alone, the accumulator of a product is its row's;
//      * ranked: a run of consecutive tiles (at most kXSpanTiles) whose output
//        is expected to fit kXRows rows: the products' rows are marked in a
//        bitmap, a prefix of its popcounts ranks the touched rows, and the
//        accumulator of a product is its row's rank, so consecutive threads
//        write consecutive output entries.  A run whose output turns out
//        larger is cut at a tile boundary.  Ranking is what lets one visit take
//        several sparse tiles: at scale 20 half of all products lie in tiles
//        of less than 8192 products and 500 output rows on average;
//      * sorted: a run of at most kXLight products is merged with the light
//        tiles that follow into a range of at most kXSort products, staged in
//        shared memory with (row, slot) keys, radix sorted by row (stable LSD,
//        7-bit digits); each run of one row is summed exactly (x_acc128).
// Columns with more than scap segments, or matrices with more than kXTMax
// tiles, visit every touched tile and look up their B entries' A segments per
// tile (tptr) instead of step 1.  Columns outside the exact window are
// appended to fb_items for the ordered kernel.
//
// Bound by instruction issue and by the latency of a visit's chain of
// barriers, not by memory (DRAM 1.4 % of peak).  Against one tile a visit with
// the segments found by searches and 24-byte accumulators behind flag bytes
// (209 instead of 498 warp instructions per 32 products), R-MAT scale 20 A*A in
// phases went from 1656 to 998 ms, all passes included (2^14: 1.94 to 1.51 ms),
// and a 30011-vertex min-plus product from 8.28 (k_numeric, warp kernels up to
// 4096 products) to 4.0 ms.
template <class SR>
__global__ void __launch_bounds__(kXThreads, 2)
    k_numeric_x(const SpgemmArgs *args, const int64_t *items, int64_t nitems, const int64_t *ccp, int64_t ccp_base,
                const int64_t *cap, int64_t *out_cnt, int32_t *overflow, int64_t *cir, void *cval_v,
                unsigned long long *work, int64_t *fb_items, unsigned long long *fb_count, XSeg *scratch_all, int64_t scap)
{
    typedef typename SR::V V;
    typedef XAcc<SR> Acc;
    constexpr bool EXACT = std::is_same<SR, PlusTimes<double>>::value;
    constexpr int NT = kXThreads, NW = NT / 32, R = kXRows;
    static_assert(kXTMax <= NT && kXSegs == 2 * NT && kXWins == NT && kXSort <= 4096 && kXSort <= 8 * NT, "block shape");
    extern __shared__ __align__(16) unsigned char xsm[];
    XSmem &sm = *reinterpret_cast<XSmem *>(xsm);
    // a sorted range reuses the accumulator (cleared again before a ranked visit)
    uint32_t *rk0 = sm.acc, *rk1 = rk0 + kXSort;                  // [kXSort] keys, sort buffer
    uint64_t *rval = reinterpret_cast<uint64_t *>(rk1 + kXSort);  // [kXSort] products
    uint32_t *rwh = reinterpret_cast<uint32_t *>(sm.rows);        // [NW][128] digit counts per warp
    static_assert(kXSort * 16 <= (int)sizeof(sm.acc) && NW * 128 * 4 <= (int)sizeof(sm.rows), "range area");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1;
    XSeg *scratch = scratch_all + (int64_t)blockIdx.x * scap;
    for (int u = tid; u < 4 * R; u += NT) sm.acc[u] = 0;
    for (int u = tid; u < kXSpanTiles * R / 32; u += NT) sm.bm[u] = 0;
    for (int u = tid; u < R / 32; u += NT) sm.term[u] = 0;
    bool dirty = false;  // the accumulator holds a sorted range's data
    bool first_item = true;
    int par = 0;  // which wsum the next prefix uses

    // block-wide exclusive prefix of v over the threads (one barrier: two
    // prefixes in a row use different sums); *tot the total
    auto block_prefix = [&](int v, int *tot) -> int {
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) sm.wsum[par][warp] = x;
        __syncthreads();
        int w = lane < NW ? sm.wsum[par][lane] : 0;
        par ^= 1;
        const int own = w;
#pragma unroll
        for (int o = 1; o < NW; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        *tot = __shfl_sync(0xffffffffu, w, NW - 1);
        return __shfl_sync(0xffffffffu, w - own, warp) + x - v;
    };
    // The chunk table.  Every thread brings two consecutive segments (start,
    // length, B value); empty ones are dropped when `compact` (elsewhere only
    // the last ones are empty).  Product p of the chunk then belongs to
    // segment win[p / 32].y - 1 + (starts up to p in win[p / 32].x), so a warp
    // finds its products' segments with one popcount and no search.  A table
    // covers rounds of kXWins windows; rounds() moves it to another one.
    // segment i holds products [p, p + len) from the round's first on
    auto set_windows = [&](int i, int p, int len) {
        if (len > 0) {
            if (p >= 0 && p < kXWins * 32) atomicOr(&sm.win[p >> 5].x, 1u << (p & 31));
            // windows that start inside this segment or right behind it
            for (int w = max(0, (p >> 5) + 1); w <= min(kXWins - 1, (p + len) >> 5); ++w) sm.win[w].y = i + 1;
        }
    };
    auto fill_table = [&](const uint32_t (&st)[2], const int (&ln)[2], const uint64_t (&bv)[2], bool compact) -> int {
        int tot, cnt = kXSegs;
        sm.win[tid] = make_uint2(0u, 0u);
        int p = block_prefix(ln[0] + ln[1], &tot);
        int c = compact ? block_prefix((ln[0] > 0) + (ln[1] > 0), &cnt) : 2 * tid;
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if (ln[u] > 0 || !compact) {
                sm.off[c] = p;
                sm.base[c] = st[u] - (uint32_t)p;
                sm.bv[c] = bv[u];
                set_windows(c, p, ln[u]);
                p += ln[u];
                ++c;
            }
        if (tid == 0) {
            sm.off[cnt] = tot;
            sm.nseg = cnt;
        }
        __syncthreads();
        return tot;
    };
    // step(q0, n) for every round of the chunk's L products (n of them from q0
    // on); `again`: the table was left at a later round.  A caller's barrier
    // ends the last round.
    auto rounds = [&](int L, bool again, auto &&step) {
        for (int q0 = 0; q0 < L; q0 += kXWins * 32) {
            if (q0 > 0 || (again && L > kXWins * 32)) {
                __syncthreads();
                sm.win[tid] = make_uint2(0u, 0u);
                __syncthreads();
                for (int i = 2 * tid; i < min(2 * tid + 2, sm.nseg); ++i)
                    set_windows(i, sm.off[i] - q0, sm.off[i + 1] - sm.off[i]);
                __syncthreads();
            }
            step(q0, min(L - q0, kXWins * 32));
        }
    };
    const unsigned le = lt | (1u << lane);
    // segment of the lane's product in window w of the round
    auto seg_of = [&](int w) -> int {
        const uint2 x = sm.win[w];
        return (int)x.y + __popc(x.x & le) - 1;
    };
    // f(b, idx, p) for the chunk's products: segment b, A position idx
    auto for_products = [&](int L, bool again, auto &&f) {
        rounds(L, again, [&](int q0, int n) {
            for (int w = warp; w * 32 < n; w += NW) {
                const int p = w * 32 + lane;
                if (p < n) {
                    const int b = seg_of(w);
                    f(b, sm.base[b] + (uint32_t)(q0 + p), q0 + p);
                }
            }
        });
    };

    for (;;) {
        if (tid == 0) {
            sm.col = next_item(work, first_item);
            if (sm.col < nitems) sm.a = args[item_pid(items[sm.col])];
        }
        __syncthreads();
        const int64_t ci = sm.col;
        if (ci >= nitems) break;
        const SpgemmArgs &a = sm.a;
        const int64_t i = item_col(items[ci]);
        const int64_t g = a.col_base + i;
        const V *bval = static_cast<const V *>(a.bval);
        const int64_t bs = a.bcp[i], be = a.bcp[i + 1];
        int out = 0;  // entries written (a column's output fits its row ids: below 2^31)
        bool over = false, bad = false;
        if (tid == 0) {
            const int64_t out0 = ccp[g - ccp_base];
            sm.bs = bs;
            sm.be = be;
            sm.oir = cir + out0;
            sm.oval = static_cast<V *>(cval_v) + out0;
            sm.lim = (int)min(cap ? cap[g] : ccp[g - ccp_base + 1] - out0, (int64_t)INT32_MAX);
        }

        for (int u = tid; u < kXTMax; u += NT) {
            sm.segcnt[u] = 0;
            sm.prodcnt[u] = 0;
        }
        // admission (exact sums): the exponent window of the column's
        // products; pos: all of them are positive; zeros: some may be zero
        bool pos = true;
        [[maybe_unused]] bool zeros = false;
        int ebase = 0;
        if constexpr (EXACT) {
            bool mixed = false, zero = false;
            int emin = 1 << 30, emax = -(1 << 30);
            for (int64_t b = bs + tid; b < be; b += NT) {
                const int32_t ae = a.aexp[a.brow[b]];
                const double bv = bval ? bval[b] : 1.0;
                x_window(ae, bv, bval != nullptr, emin, emax);
                mixed |= (ae & kXMixed) || !(bv > 0.0);
                zero |= (ae & kXZero) || bv == 0.0;
            }
            emin = __reduce_min_sync(0xffffffffu, emin);
            emax = __reduce_max_sync(0xffffffffu, emax);
            zero = __any_sync(0xffffffffu, zero);
            if (lane == 0) {
                sm.emin[warp] = emin;
                sm.emax[warp] = emax;
                sm.wzero[warp] = zero;
            }
            pos = !__syncthreads_or(mixed);
            zeros = __any_sync(0xffffffffu, sm.wzero[lane & (NW - 1)]);
            ebase = __reduce_min_sync(0xffffffffu, sm.emin[lane & (NW - 1)]);
            const int etop = __reduce_max_sync(0xffffffffu, sm.emax[lane & (NW - 1)]);
            if (!x_admit(ebase, etop, be - bs)) {
                if (tid == 0) fb_items[atomicAdd(fb_count, 1ull)] = items[ci];
                __syncthreads();  // sm.col / sm.a / sm.emin reuse
                continue;
            }
            if (tid == 0) sm.ebase = ebase;  // read behind the barriers of the chunk tables
        } else {
            __syncthreads();
        }

        // ---- a ranked visit's steps.  Rows are relative to the visit's first row row0.
        auto mark = [&](int L, int row0) {
            const int32_t *arow = sm.a.arow;
            rounds(L, false, [&](int q0, int n) {
                for (int w = warp; w * 32 < n; w += 2 * NW) {  // two windows at a time
                    const int p = w * 32 + lane, p2 = p + NW * 32;
                    int r = -1, r2 = -1;
                    if (p < n) r = arow[sm.base[seg_of(w)] + (uint32_t)(q0 + p)] - row0;
                    if (p2 < n) r2 = arow[sm.base[seg_of(w + NW)] + (uint32_t)(q0 + p2)] - row0;
                    if (r >= 0) atomicOr(&sm.bm[r >> 5], 1u << (r & 31));
                    if (r2 >= 0) atomicOr(&sm.bm[r2 >> 5], 1u << (r2 & 31));
                }
            });
        };
        // Products added into the accumulators: of their row's rank, or of
        // the row itself (DIRECT, one tile: the row is marked here as well).
        // The loads of the warp's next window are issued before the current
        // window's atomics.  SIGN: 0 the products are positive, 1 of either
        // sign, 2 some may be zero: then `term` marks the accumulators that got
        // another term than -0.0, which alone leaves an exact zero -0.0.
        auto accumulate_as = [&](int L, int row0, auto sign_t, auto direct_t) {
            [[maybe_unused]] constexpr int SIGN = decltype(sign_t)::value;
            constexpr bool DIRECT = decltype(direct_t)::value;
            const int32_t *arow = sm.a.arow;
            const V *aval = static_cast<const V *>(sm.a.aval);
            [[maybe_unused]] const int ebase = sm.ebase;
            rounds(L, true, [&](int q0, int n) {
                int r_n = -1;
                V a_n = SR::one(), b_n = SR::one();
                auto load = [&](int w) {
                    const int p = w * 32 + lane;
                    r_n = -1;
                    if (p < n) {
                        const int b = seg_of(w);
                        const uint32_t idx = sm.base[b] + (uint32_t)(q0 + p);
                        r_n = arow[idx] - row0;
                        a_n = aval ? aval[idx] : SR::one();
                        b_n = x_from<V>(sm.bv[b]);
                    }
                };
                load(warp);
                for (int w = warp; w * 32 < n; w += NW) {
                    const int r = r_n;
                    const V av = a_n, bv = b_n;
                    load(w + NW);
                    if (r >= 0) {
                        const V prod = SR::mul(av, bv);
                        int at = r;
                        if (DIRECT) {
                            atomicOr(&sm.bm[r >> 5], 1u << (r & 31));
                        } else {
                            at = sm.pre[r >> 5] + __popc(sm.bm[r >> 5] & ((1u << (r & 31)) - 1));
                            sm.rows[at] = (uint16_t)r;  // every product of the row writes the same
                        }
                        if constexpr (EXACT) {
                            const uint64_t bits = (uint64_t)__double_as_longlong(prod);
                            if (SIGN == 2 && bits != 1ull << 63) {
                                const uint32_t bit = 1u << (at & 31);
                                if (!(sm.term[at >> 5] & bit)) atomicOr(&sm.term[at >> 5], bit);
                            }
                            if ((SIGN < 2 || (bits << 1) != 0) && !x_add128<SIGN == 0>(sm.acc + at, R, bits, ebase))
                                bad = true;
                        } else if (!Acc::add(sm.acc, R, at, prod)) {
                            bad = true;
                        }
                    }
                }
            });
        };
        auto accumulate = [&](int L, int row0, auto direct_t) {
            if (!EXACT || pos)
                accumulate_as(L, row0, std::integral_constant<int, 0>{}, direct_t);
            else if (!zeros)
                accumulate_as(L, row0, std::integral_constant<int, EXACT ? 1 : 0>{}, direct_t);
            else
                accumulate_as(L, row0, std::integral_constant<int, EXACT ? 2 : 0>{}, direct_t);
        };
        // ranks of the touched rows among the first nw bitmap words (at most
        // 4 per thread); *before(t) is left in pre[]; returns the total
        auto rank_rows = [&](int nw) -> int {
            constexpr int PER = kXSpanTiles * R / 32 / NT;
            const int per = (nw + NT - 1) / NT;  // block-uniform
            int pc[PER], sum = 0;
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int w = tid * per + u;
                pc[u] = (u < per && w < nw) ? __popc(sm.bm[w]) : 0;
                sum += pc[u];
            }
            int tot;
            int run = block_prefix(sum, &tot);
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int w = tid * per + u;
                if (u < per && w < nw) sm.pre[w] = (uint16_t)run;
                run += pc[u];
            }
            __syncthreads();
            return tot;
        };
        // accumulator `at` (row row0 + r) rounded and written as output entry q of the visit, and cleared
        auto write_one = [&](int at, int q, int r, int row0) {
            V v;
            if constexpr (EXACT) {
                uint32_t *w = sm.acc + at;
                const uint64_t lo = w[0] | ((uint64_t)w[R] << 32), hi = w[2 * R] | ((uint64_t)w[3 * R] << 32);
                w[0] = 0;
                w[R] = 0;
                w[2 * R] = 0;
                w[3 * R] = 0;
                v = x_round(hi, lo, !zeros || (sm.term[at >> 5] >> (at & 31) & 1) ? 2 : 0, sm.ebase);
            } else {
                v = Acc::take(sm.acc, R, at);
            }
            q += out;
            if (q < sm.lim) {
                sm.oir[q] = row0 + r;
                static_cast<V *>(sm.oval)[q] = v;
            } else {
                over = true;
            }
        };
        auto end_visit = [&](int n) {
            __syncthreads();
            if (EXACT && zeros)  // block-uniform; marked again only after another visit's barriers
                for (int w = tid; w < R / 32; w += NT) sm.term[w] = 0;
            out += n;
        };
        // a ranked visit's n entries; the bitmap's first nw words are cleared
        auto write_ranks = [&](int n, int nw, int row0) {
            for (int q = tid; q < n; q += NT) write_one(q, q, sm.rows[q], row0);
            for (int w = tid; w < nw; w += NT) sm.bm[w] = 0;
            end_visit(n);
        };
        // a direct visit's entries: a warp per bitmap word
        auto write_direct = [&](int nw, int row0) {
            const int n = rank_rows(nw);
            for (int w = warp; w < nw; w += NW) {
                const uint32_t x = sm.bm[w];
                if ((x >> lane) & 1) write_one(w * 32 + lane, sm.pre[w] + __popc(x & lt), w * 32 + lane, row0);
                __syncwarp();
                if (lane == 0) sm.bm[w] = 0;
            }
            end_visit(n);
        };
        auto clean = [&]() {
            if (dirty) {
                for (int u = tid; u < 4 * R; u += NT) sm.acc[u] = 0;
                dirty = false;
                __syncthreads();
            }
        };

        // ------------------------------------------------ 1. bucketing
        bool bucketed = a.T <= kXTMax && a.ktl_ptr != nullptr;  // block-uniform
        if (bucketed) {
            // pass 0 counts, pass 1 scatters: the (entry, tile) pairs of a
            // chunk of entries are flattened over the warps like products
            for (int pass = 0; pass < 2; ++pass) {
                for (int64_t cb = bs; cb < be; cb += kXSegs) {
                    uint32_t st[2];
                    int ln[2];
                    uint64_t en[2];  // the entry, carried in the table's value slot
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int64_t e = cb + 2 * tid + u;
                        st[u] = 0;
                        ln[u] = 0;
                        en[u] = (uint64_t)(e - bs);
                        if (e < be) {
                            const int k = a.brow[e];
                            const int64_t p0 = a.ktl_ptr[k];
                            st[u] = (uint32_t)p0;
                            ln[u] = (int)(a.ktl_ptr[k + 1] - p0) - 1;  // touched tiles (the end marker excluded)
                        }
                    }
                    const int L = fill_table(st, ln, en, true);
                    for_products(L, false, [&](int b, uint32_t q, int) {
                        const int t = a.ktl_tile[q];
                        const uint32_t s0 = a.ktl_start[q];
                        const int len = (int)(a.ktl_start[q + 1] - s0);
                        if (pass == 0) {
                            atomicAdd(&sm.segcnt[t], 1);
                            atomicAdd(&sm.prodcnt[t], len);
                        } else {
                            const int pos = atomicAdd(&sm.tend[t], 1);
                            scratch[pos] = XSeg{s0, (uint32_t)len, (uint32_t)sm.bv[b]};
                        }
                    });
                    __syncthreads();
                }
                if (pass == 0) {
                    // tile offsets; a column with too many segments is not bucketed
                    int tot;
                    const int ex = block_prefix(tid < a.T ? sm.segcnt[tid] : 0, &tot);
                    if (tot > scap) {
                        bucketed = false;  // block-uniform: tot is
                        break;
                    }
                    if (tid < a.T) sm.tend[tid] = ex;
                    __syncthreads();
                }
            }
            // tend[t] is now the end of tile t's segments
        }

        // segments [c0, min(c0 + kXSegs, se)) of the scratch: this thread's two
        auto fetch = [&](XSeg (&sg)[2], int c0, int se) {
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int c = c0 + 2 * tid + u;
                sg[u] = c < se ? scratch[c] : XSeg{0, 0, 0};
            }
        };
        auto load_bucket = [&](const XSeg (&sg)[2]) -> int {
            const uint32_t st[2] = {sg[0].start, sg[1].start};
            const int ln[2] = {(int)sg[0].len, (int)sg[1].len};
            uint64_t bv[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const V *b = static_cast<const V *>(sm.a.bval);
                bv[u] = x_bits<V>(b ? b[sm.bs + sg[u].e] : SR::one());
            }
            return fill_table(st, ln, bv, false);
        };
        // The next run from tile t on (lanes hold one tile each): t its first
        // touched tile (a.T: none), t1 its end.  Of p products over R rows
        // about p / (1 + p / R) rows are expected.
        int t = 0, t1 = 0, segs = 0, prods = 0;
        bool direct = false;
        auto next_run = [&]() {
            for (; t < a.T; t += 32) {
                const unsigned m = __ballot_sync(0xffffffffu, t + lane < a.T && sm.segcnt[t + lane] > 0);
                if (m) {
                    t += __ffs(m) - 1;
                    break;
                }
            }
            if (t >= a.T) {
                t = t1 = a.T;
                return;
            }
            const int u = t + lane;
            const bool in = lane < kXSpanTiles && u < a.T;
            int s = in ? sm.segcnt[u] : 0, p = in ? sm.prodcnt[u] : 0;
            const bool some = s > 0, heavy = p > kXDirect;
            int e = p >= 8 * R ? R : (int)__fdividef((float)p, 1.0f + (float)p * (1.0f / R));
#pragma unroll
            for (int o = 1; o < kXSpanTiles; o <<= 1) {
                const int se = __shfl_up_sync(0xffffffffu, s, o), pe = __shfl_up_sync(0xffffffffu, p, o),
                          ee = __shfl_up_sync(0xffffffffu, e, o);
                if (lane >= o) {
                    s += se;
                    p += pe;
                    e += ee;
                }
            }
            const bool fits = in && !heavy && e <= R && s <= kXSegs && p <= kXWins * 32;
            const unsigned tm = __ballot_sync(0xffffffffu, some);
            unsigned ok = __ballot_sync(0xffffffffu, fits);
            direct = !(ok & 1);  // the first tile does not fit a ranked visit: a visit of its own
            if (direct) ok = 1;
            // tiles before the first that does not fit, less untouched ones at the end
            const unsigned run = tm & ((ok + 1) & ~ok) - 1;
            const int last = 31 - __clz(run);
            t1 = t + last + 1;
            segs = __shfl_sync(0xffffffffu, s, last);
            prods = __shfl_sync(0xffffffffu, p, last);
        };

        if (bucketed) {
            // -------------------------------------------- 2. visits in row order
            XSeg sg[2];
            next_run();
            while (t < a.T) {
                const int row0 = t * R;
                const int sb = sm.tend[t] - sm.segcnt[t];
                if (direct || prods > kXLight) {
                    clean();
                    int nw = (int)((min(t1 * (int64_t)R, a.m) - row0 + 31) >> 5);
                    int n = 0;
                    if (direct) {
                        for (int c0 = sb; c0 < sb + segs; c0 += kXSegs) {
                            fetch(sg, c0, sb + segs);
                            if (c0 > sb) __syncthreads();
                            accumulate(load_bucket(sg), row0, std::true_type{});
                        }
                    } else {
                        fetch(sg, sb, sb + segs);
                        int L = load_bucket(sg);
                        mark(L, row0);
                        __syncthreads();
                        n = rank_rows(nw);
                        if (n > R) {
                            // too many rows: keep the first tiles that fit
                            while (n > R) {
                                --t1;
                                L -= sm.prodcnt[t1];
                                n = sm.pre[(t1 - t) * (R / 32)];
                            }
                            for (int w = (t1 - t) * (R / 32) + tid; w < nw; w += NT) sm.bm[w] = 0;
                            nw = (t1 - t) * (R / 32);
                        }
                        accumulate(L, row0, std::false_type{});
                    }
                    if (tid == 0) atomicAdd(&work[t1 - t > 1 ? 2 : 1], 1ull);  // visits of one tile / of a run
                    __syncthreads();
                    if (direct) {
                        write_direct(nw, row0);
                    } else {
                        write_ranks(n, nw, row0);
                    }
                    t = t1;
                    next_run();
                } else {
                    // sorted range of light tiles t .. t1 (at most kXSort products)
                    t1 = t;
                    prods = sm.prodcnt[t];
                    // (more segments are more products, whose count may have passed 2^31)
                    while (t1 + 1 < a.T && (sm.segcnt[t1 + 1] == 0 ||
                                            (sm.segcnt[t1 + 1] <= kXLight && sm.prodcnt[t1 + 1] <= kXLight &&
                                             prods + sm.prodcnt[t1 + 1] <= kXSort))) {
                        ++t1;
                        prods += sm.prodcnt[t1];
                    }
                    while (sm.segcnt[t1] == 0) --t1;  // end on a touched tile
                    const int span_rows = (t1 - t + 1) * R;  // <= 2^20
                    const int se = sm.tend[t1];
                    dirty = true;
                    // stage: key = (row - row0) << 12 | slot, value = the product
                    int pbase = 0;
                    for (int c0 = sb; c0 < se; c0 += kXSegs) {
                        fetch(sg, c0, se);
                        const int L = load_bucket(sg);
                        const int32_t *arow = sm.a.arow;
                        const V *aval = static_cast<const V *>(sm.a.aval);
                        for_products(L, false, [&](int b, uint32_t idx, int p) {
                            const int slot = pbase + p;
                            rk0[slot] = ((uint32_t)(arow[idx] - row0) << 12) | (uint32_t)slot;
                            rval[slot] = x_bits<V>(SR::mul(aval ? aval[idx] : SR::one(), x_from<V>(sm.bv[b])));
                        });
                        pbase += L;
                        __syncthreads();  // chunk table reuse
                    }
                    if (tid == 0) atomicAdd(&work[2], 1ull);
                    // stable LSD radix sort of the keys by row, 7-bit digits:
                    // warp w owns a contiguous run of keys, counts its digits,
                    // the (digit, warp) counts are scanned digit-major, and
                    // each warp scatters its keys in order (rank inside a
                    // 32-key window from seven ballots)
                    const int rbits = span_rows > 1 ? 32 - __clz(span_rows - 1) : 1;
                    uint32_t *src = rk0, *dst = rk1;
                    const int per = (((prods + NW - 1) / NW) + 31) & ~31;
                    const int k0 = min(prods, warp * per), k1 = min(prods, k0 + per);
                    uint32_t *wh = rwh + warp * 128;
                    for (int shift = 12; shift < 12 + rbits; shift += 7) {
                        for (int u = lane; u < 128; u += 32) wh[u] = 0;
                        __syncwarp();
                        for (int u = k0 + lane; u < k1; u += 32) atomicAdd(&wh[(src[u] >> shift) & 127], 1u);
                        __syncthreads();
                        {  // exclusive scan over (digit, warp), digit-major
                            constexpr int PER = NW * 128 / NT;
                            int loc[PER], sum = 0;
#pragma unroll
                            for (int j = 0; j < PER; ++j) {
                                const int idx = tid * PER + j, d = idx / NW, w = idx - d * NW;
                                loc[j] = (int)rwh[w * 128 + d];
                                sum += loc[j];
                            }
                            int tot;
                            int run = block_prefix(sum, &tot);
#pragma unroll
                            for (int j = 0; j < PER; ++j) {
                                const int idx = tid * PER + j, d = idx / NW, w = idx - d * NW;
                                rwh[w * 128 + d] = (uint32_t)run;
                                run += loc[j];
                            }
                        }
                        __syncthreads();
                        for (int b0 = k0; b0 < k1; b0 += 32) {
                            const int u = b0 + lane;
                            const bool act = u < k1;
                            const uint32_t key = act ? src[u] : 0u;
                            const int d = (int)((key >> shift) & 127);
                            unsigned same = __ballot_sync(0xffffffffu, act);
#pragma unroll
                            for (int bit = 0; bit < 7; ++bit) {
                                const unsigned bb = __ballot_sync(0xffffffffu, act && ((d >> bit) & 1));
                                same &= ((d >> bit) & 1) ? bb : ~bb;
                            }
                            const int rank = __popc(same & lt);
                            if (act) dst[wh[d] + rank] = key;
                            __syncwarp();
                            if (act && rank == 0) wh[d] += __popc(same);
                            __syncwarp();
                        }
                        __syncthreads();
                        uint32_t *tmp = src;
                        src = dst;
                        dst = tmp;
                    }
                    // runs of one row, one sorted key per thread and round:
                    // the thread holding a run's first key sums the run
                    // exactly (runs are short: a range's rows rarely repeat)
                    // and writes it; output positions from a block prefix of
                    // the run heads, so consecutive threads write
                    // consecutive entries
                    for (int u0 = 0; u0 < prods; u0 += NT) {
                        const int u = u0 + tid;
                        const bool act = u < prods;
                        const uint32_t key = act ? src[u] : 0u;
                        const bool head = act && (u == 0 || (src[u - 1] >> 12) != (key >> 12));
                        int tot;
                        const int q = out + block_prefix(head ? 1 : 0, &tot);
                        if (head) {
                            const uint32_t row = key >> 12;
                            V val;
                            if constexpr (EXACT) {
                                uint64_t hi = 0, lo = 0;
                                uint32_t fl = 0;
                                for (int v = u; v < prods; ++v) {
                                    const uint32_t kv = src[v];
                                    if ((kv >> 12) != row) break;
                                    if (!x_acc128(hi, lo, fl, x_from<double>(rval[kv & 4095]), ebase)) bad = true;
                                }
                                val = x_round(hi, lo, fl, ebase);
                            } else {  // any order would do
                                val = x_from<V>(rval[key & 4095]);
                                for (int v = u + 1; v < prods && (src[v] >> 12) == row; ++v)
                                    val = SR::add(x_from<V>(rval[src[v] & 4095]), val);
                                if constexpr (std::is_same<SR, MinPlus<double>>::value) {
                                    for (int v = u; v < prods && (src[v] >> 12) == row; ++v) {
                                        const uint64_t pb = rval[src[v] & 4095];
                                        if (pb == 1ull << 63 || x_from<double>(pb) != x_from<double>(pb)) bad = true;
                                    }
                                }
                            }
                            if (q < sm.lim) {
                                sm.oir[q] = (int64_t)row0 + (int64_t)row;
                                static_cast<V *>(sm.oval)[q] = val;
                            } else {
                                over = true;
                            }
                        }
                        out += tot;
                    }
                    __syncthreads();
                    t = t1 + 1;
                    next_run();
                }
            }
        } else {
            // ------------------------- enumeration mode: per tile, all entries
            clean();
            int mwi = 0;
            uint64_t msk = a.tmask[i * a.mask_words];
            auto next_tile = [&]() -> int {
                while (msk == 0) {
                    if (++mwi >= a.mask_words) return -1;
                    msk = a.tmask[i * a.mask_words + mwi];
                }
                const int tt = mwi * 64 + __ffsll((long long)msk) - 1;
                msk &= msk - 1;
                return tt;
            };
            for (t = next_tile(); t >= 0; t = next_tile()) {
                const int row0 = t * R;
                const int nw = (int)((min((int64_t)(t + 1) * R, a.m) - row0 + 31) >> 5);
                for (int64_t cb = bs; cb < be; cb += kXSegs) {
                    uint32_t st[2];
                    int ln[2];
                    uint64_t bv[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int64_t e = cb + 2 * tid + u;
                        st[u] = 0;
                        ln[u] = 0;
                        bv[u] = x_bits<V>(SR::one());
                        if (e < be) {
                            const uint32_t *tp = a.tptr + (int64_t)a.brow[e] * (a.T + 1);
                            st[u] = tp[t];
                            ln[u] = (int)(tp[t + 1] - st[u]);
                            if (bval) bv[u] = x_bits<V>(bval[e]);
                        }
                    }
                    accumulate(fill_table(st, ln, bv, true), row0, std::true_type{});
                    __syncthreads();
                }
                if (tid == 0) atomicAdd(&work[1], 1ull);
                write_direct(nw, row0);
            }
        }
        over = __syncthreads_or(over);
        bad = __syncthreads_or(bad);
        if (tid == 0) {
            if (out_cnt) out_cnt[g] = out;
            if (over) {
                if (overflow)
                    overflow[g] = 1;
                else
                    atomicOr(a.err, 128);  // exact sizing: counts disagree
            }
            if (bad && EXACT) atomicOr(a.err, 512);  // a product outside the admitted window
            if (bad && !EXACT) fb_items[atomicAdd(fb_count, 1ull)] = items[ci];  // XAcc: the ordered kernel's
        }
    }
}

}  // namespace gbc
