// Ordered SpGEMM columns whose rows are owned by warps (included by spgemm.cu).
//
// A column's output is the left fold acc = add(mrhs, acc) over its B entries
// in order (mtSpGEMM.h:396-412).  Where a column is dense enough that every B
// entry brings several products to every 1/T2 of the rows, a warp takes one
// such range of rows, keeps their accumulators in shared memory and walks the
// B entries in order: a segment of one A column has distinct rows, so its
// products are folded lane by lane with plain loads and stores -- no
// partition of products to owners, no atomics, no barriers until the column's
// ranges are written.
//
// Bound by issue and the latency of short segments (about 28 of a window's 32
// lanes hold a product in an MCL loop).  The ordered kernel k_numeric, which
// stages and partitions every product, took 381 ms where this takes 165 (MCL
// loop on 20000 vertices, its dense iterations).
//
// The ranges split the rows evenly by a weight of one half each of the rows
// and of A's entries in them, so that skewed rows do not leave one warp with
// the work, and no range exceeds 2 m / T2 + 1 rows.
#pragma once

namespace gbc {

// Four warps a block: the barriers that order a column's ranges in the output
// hold up few warps (an MCL loop takes 303 ms with eight, 292 with sixteen and
// 280 with four).
constexpr int kOwnThreads = 128;
constexpr int kOwnWarps = kOwnThreads / 32;
constexpr int kOwnRanges = 128;             // ranges at most
constexpr int64_t kOwnTable = 1ll << 28;    // pointers of a product's range table, at most
constexpr int kOwnSmem = 6656 * kOwnWarps;  // accumulators and marks of a block (32 warps per SM)

// Products per B entry and range from which a column is dense enough.  Below,
// windows are mostly empty: 8-byte values (measured with min-plus, which
// k_numeric_x has taken over since) on a 30011-vertex R-MAT took 8.2 ms with 16,
// 8.6 with 8 and 14.6 with 4 (k_numeric alone 8.3); fp32 ranges are
// nearly twice as wide, an MCL loop takes 263 ms with 8, 280 with 16, 450 without.
__host__ __device__ constexpr int own_min(int vsize) { return vsize <= 4 ? 8 : 16; }

// Rows of a range at most, for values of vsize bytes (a mark byte beside each).
__host__ __device__ constexpr int own_rows(int vsize)
{
    return (kOwnSmem / kOwnWarps / (vsize + 1)) / 32 * 32 < 2048 ? (kOwnSmem / kOwnWarps / (vsize + 1)) / 32 * 32 : 2048;
}

// Ranges for m rows: a whole number per warp; 0 where the rows are too many.
inline int own_ranges(int64_t m, int64_t ncol, int vsize)
{
    const int64_t per = own_rows(vsize) - 2;
    const int64_t t = ((2 * m + per - 1) / per + kOwnWarps - 1) / kOwnWarps * kOwnWarps;
    return t <= kOwnRanges && ncol * (t + 1) <= kOwnTable ? (int)t : 0;
}

static __global__ void k_own_count(int64_t nnz, const int32_t *arow, unsigned long long *rowcnt)
{
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < nnz) atomicAdd(&rowcnt[arow[i]], 1ull);
}

static __global__ void k_own_weight(int64_t m, int64_t nnz, int64_t *rowcnt)
{
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r < m) rowcnt[r] = rowcnt[r] * m + nnz;
}

// Range of every row from the weights' prefix (total 2 m nnz), and the first row of every range.
static __global__ void k_own_bounds(int64_t m, int64_t nnz, int T2, const int64_t *prefix, uint8_t *range, int32_t *rb)
{
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r >= m) return;
    const int64_t total = 2 * m * nnz;
    auto of = [&](int64_t row) { return (int)min((int64_t)(T2 - 1), prefix[row] / ((total + T2 - 1) / T2)); };
    const int t = of(r), before = r > 0 ? of(r - 1) : -1;
    range[r] = (uint8_t)t;
    for (int u = before + 1; u <= t; ++u) rb[u] = (int32_t)r;
    if (r == m - 1)
        for (int u = t + 1; u <= T2; ++u) rb[u] = (int32_t)m;
}

// optr[k * (T2 + 1) + t]: first position of column k of A in range t or later.
static __global__ void k_own_ptr(int64_t ncol, const int64_t *acp, const int32_t *arow, const uint8_t *range, int T2,
                                 uint32_t *optr)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t k = warp; k < ncol; k += nwarps) {
        uint32_t *tp = optr + k * (T2 + 1);
        const int64_t s = acp[k], e = acp[k + 1];
        for (int64_t p = s + lane; p < e; p += 32) {
            const int t = range[arow[p]], before = p > s ? range[arow[p - 1]] : -1;
            for (int u = before + 1; u <= t; ++u) tp[u] = (uint32_t)p;
        }
        const int last = e > s ? range[arow[e - 1]] : -1;
        for (int u = last + 1 + lane; u <= T2; u += 32) tp[u] = (uint32_t)e;
    }
}

template <class SR>
__global__ void __launch_bounds__(kOwnThreads, 1024 / kOwnThreads) k_numeric_own(const SpgemmArgs *args, const int64_t *items,
                                                                int64_t nitems, const int64_t *ccp, int64_t ccp_base,
                                                                const int64_t *cap, int64_t *out_cnt,
                                                                int32_t *overflow, int64_t *cir, void *cval_v,
                                                                unsigned long long *work)
{
    typedef typename SR::V V;
    constexpr int RC = own_rows(sizeof(V)), NW = kOwnWarps, U = 2;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int64_t s_col;
    __shared__ SpgemmArgs sa;
    __shared__ int s_cnt[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1;
    V *acc = reinterpret_cast<V *>(smem) + warp * RC;
    uint8_t *tag = smem + (size_t)NW * RC * sizeof(V) + warp * RC;
    V *cval = static_cast<V *>(cval_v);
    for (int r = lane; r < RC; r += 32) {
        acc[r] = SR::zero();
        tag[r] = 0;
    }
    __syncwarp();
    bool first_item = true;
    for (;;) {
        if (tid == 0) {
            s_col = next_item(work, first_item);
            if (s_col < nitems) sa = args[item_pid(items[s_col])];
        }
        __syncthreads();
        const int64_t ci = s_col;
        if (ci >= nitems) break;
        const int64_t i = item_col(items[ci]), g = sa.col_base + i;
        const int T2 = sa.own_T;
        const uint32_t *optr = sa.own_ptr;
        const int32_t *arow = sa.arow, *brow = sa.brow, *rb = sa.own_rb;
        const V *aval = static_cast<const V *>(sa.aval), *bval = static_cast<const V *>(sa.bval);
        const int64_t bs = sa.bcp[i], be = sa.bcp[i + 1];
        const int64_t out0 = ccp[g - ccp_base];
        const int64_t lim = cap ? out0 + cap[g] : ccp[g - ccp_base + 1];
        int64_t out = out0;
        bool over = false;
        for (int t0 = 0; t0 < T2; t0 += NW) {
            const int t = t0 + warp;
            const int row0 = rb[t], rows = rb[t + 1] - row0;
            // B entries in order, 32 at a time, one per lane; the next 32 are loaded ahead
            int kn = bs + lane < be ? brow[bs + lane] : -1;
            for (int64_t cb = bs; cb < be && rows > 0; cb += 32) {
                const int k = kn;
                uint32_t s = 0, e = 0;
                V bv = SR::one();
                if (k >= 0) {
                    const uint32_t *tp = optr + (int64_t)k * (T2 + 1) + t;
                    s = tp[0];
                    e = tp[1];
                    if (bval) bv = bval[cb + lane];
                }
                kn = cb + 32 + lane < be ? brow[cb + 32 + lane] : -1;
                // windows of 32 products: incl, the windows up to and with this lane's entry
                const int nwin = (int)((e - s + 31) >> 5);
                int incl = nwin;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                const int W = __shfl_sync(0xffffffffu, incl, 31);
                const uint32_t first = s - (uint32_t)(incl - nwin) * 32;  // position of window 0's lane 0 as this entry sees it
                // U windows are loaded while the U before them are folded
                int row_n[U];
                V av_n[U], bb_n[U];
                auto load = [&](int q0) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        row_n[u] = -1;
                        const int q = q0 + u;
                        if (q < W) {  // warp-uniform
                            const int j = __popc(__ballot_sync(0xffffffffu, incl <= q));
                            const uint32_t p = __shfl_sync(0xffffffffu, first, j) + (uint32_t)(q * 32 + lane);
                            bb_n[u] = __shfl_sync(0xffffffffu, bv, j);
                            if (p < __shfl_sync(0xffffffffu, e, j)) {
                                row_n[u] = arow[p] - row0;
                                av_n[u] = aval ? aval[p] : SR::one();
                            }
                        }
                    }
                };
                load(0);
                for (int q0 = 0; q0 < W; q0 += U) {
                    int row[U];
                    V av[U], bb[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        row[u] = row_n[u];
                        av[u] = av_n[u];
                        bb[u] = bb_n[u];
                    }
                    load(q0 + U);
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (row[u] >= 0) {
                            acc[row[u]] = SR::add(SR::mul(av[u], bb[u]), acc[row[u]]);
                            tag[row[u]] = 1;
                        }
                        __syncwarp();  // the next window's lanes see this one's sums
                    }
                }
            }
            int c = 0;
            for (int r = lane; r < rows; r += 32) c += tag[r];
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane == 0) s_cnt[warp] = c;
            __syncthreads();
            int before = 0, tot = 0;
#pragma unroll
            for (int u = 0; u < NW; ++u) {
                before += u < warp ? s_cnt[u] : 0;
                tot += s_cnt[u];
            }
            int64_t pos = out + before;
            for (int r0 = 0; r0 < rows; r0 += 32) {
                const int r = r0 + lane;
                const bool f = r < rows && tag[r];
                const unsigned m = __ballot_sync(0xffffffffu, f);
                if (f) {
                    const int64_t q = pos + __popc(m & lt);
                    if (q < lim) {
                        cir[q] = (int64_t)row0 + r;
                        cval[q] = acc[r];
                    } else {
                        over = true;  // never write past the column's range
                    }
                    acc[r] = SR::zero();
                    tag[r] = 0;
                }
                pos += __popc(m);
            }
            out += tot;
            __syncthreads();
        }
        over = __syncthreads_or(over);
        if (tid == 0) {
            if (out_cnt) out_cnt[g] = out - out0;
            if (over) {
                if (overflow)
                    overflow[g] = 1;
                else
                    atomicOr(sa.err, 128);  // exact sizing: counts disagree
            }
        }
    }
}

}  // namespace gbc
