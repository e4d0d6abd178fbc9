// Sparse matrix x sparse vector over the semirings of the reference's other
// SpMXSpV instantiations (the overload set of SpImpl.h:49-142):
//   Select2ndMin / SelectMin  y(r) = min of the x values whose column hits r
//                             (SpMXSpV_Bucket, SpImpl.cpp:389-699);
//   Select2nd (bool A)        y(r) = the x value of the LAST column, in
//                             ascending column order, that hits r -- add keeps
//                             its second argument (Semirings.h:144-163) and the
//                             boolean SPA loops of SpImpl.cpp:167-328 visit the
//                             columns in ascending order; TopDownBFS reaches it
//                             through BFSFriends.h:198-207;
//   SelectMax (bool A)        y(r) = max of the x values (Semirings.h:192-210);
//   PlusTimes (f64/f32/i64)   y(r) = sum over hitting columns c of A(r,c)*x(c),
//                             folded left in ascending column order: the
//                             first product is stored, later ones are added,
//                             as the SPA of SpMXSpV_Bucket does (bit-exact).
// A plan holds A on the device once (CSC, and for PlusTimes also row-major),
// with its scratch, so repeated multiplies by one matrix copy only vectors.
//
// GPU form.  The order-independent semirings push: blocks take the vector's
// columns in chunks, flatten their row segments and do one 64-bit atomicMax
// per product into a per-row key (min through the complemented order-
// preserving flip, Select2nd through (column << 32 | vector position)),
// marking a touched-row bitmap.  Rows come out ascending from a popcount
// scan of the bitmap.  PlusTimes pushes the marks and counts the products per
// row; the same scan then places every row's products.  A second push writes
// them (entry, product) to their row's place in any order, and each row folds
// its own in the order of the entries, which is ascending column order (and the
// stored order where a column holds a row twice): in a thread up to kSxThread
// products, in a warp up to 32, in a block up to kSxSort.  Longer rows, all rows of a vector
// that brings more than 1/kSxPullShare of the matrix, and all rows of a matrix of
// fewer than kSxPushNnz entries are pulled instead:
// a warp walks the row's row-major entries (ascending column), tests them
// against a dense column -> vector position map and folds the hits in order.
// (One window of 32 entries at a time, the longest pulled row took 0.59 of 0.69 ms
// over 2000 entries of 2^18; with eight in flight the call is about as fast as pushed.)
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "gbc_internal.cuh"
#include "spgemm_kernels.cuh"
#include "spmv_plan.cuh"

namespace gbc {

enum { SX_SELECT2NDMIN = 0, SX_SELECT2ND = 1, SX_SELECTMAX = 2, SX_PLUSTIMES = 3 };

constexpr int kSxThreads = 256;
constexpr unsigned long long kSign = 0x8000000000000000ull;

struct SpmspvPlan {
    Context *ctx = nullptr;
    int64_t m = 0, n = 0, nnz = 0;
    int vt = 0;
    int64_t *cp = nullptr;   // [n+1] dense column pointers
    int32_t *row = nullptr;  // [nnz]
    void *cval = nullptr;    // [nnz] values, column-major (numeric value types only)
    SpmvPlan rm;             // row-major form (numeric value types only)
    bool have_rm = false;
    // scratch kept between calls: every call leaves it as it found it (SxRestore)
    unsigned long long *spa = nullptr;  // [m] per-row key, 0 when untouched
    uint32_t *mark = nullptr;           // [words] touched rows
    int64_t *pos = nullptr;             // [words + 1] output offsets
    int32_t *xpos = nullptr;            // [n] 1 + vector position of a column, 0 when absent
    int32_t *err = nullptr;
    unsigned long long *work = nullptr;
    int64_t words = 0;
};

// Per stored column: dense column counts, checks, int32 rows.
__global__ void k_sx_prep(int64_t nzc, int64_t m, int64_t n, int64_t nnz, const int64_t *cp, const int64_t *jc,
                          const int64_t *ir, int64_t *cnt, int32_t *row, int32_t *err)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t i = warp; i < nzc; i += nwarps) {
        const int64_t s = cp[i], e = cp[i + 1];
        const int64_t c = jc ? jc[i] : i;
        const bool bad = e < s || s < 0 || e > nnz || (i == 0 && s != 0) || (i == nzc - 1 && e != nnz) || c < 0 ||
                         c >= n || (jc && i > 0 && jc[i - 1] >= c);
        if (bad) {
            if (lane == 0) atomicOr(err, 1);
            continue;
        }
        if (lane == 0) cnt[c] = e - s;
        for (int64_t p = s + lane; p < e; p += 32) {
            int64_t r = ir[p];
            if (r < 0 || r >= m) {
                atomicOr(err, 2);
                r = 0;
            }
            row[p] = (int32_t)r;
        }
    }
}

template <typename V>
__global__ void k_sx_ones(int64_t n, V *v)
{
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) v[i] = V(1);
}

// Vector positions of the columns; flags columns out of range (1) and
// repeated columns (2).
__global__ void k_sx_xpos(int64_t nx, const int32_t *xind, int64_t n, int32_t *xpos, int32_t *err)
{
    const int64_t f = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (f >= nx) return;
    const int32_t c = xind[f];
    if (c < 0 || c >= n) {
        atomicOr(err, 1);
        return;
    }
    if (atomicExch(&xpos[c], (int32_t)(f + 1)) != 0) atomicOr(err, 2);
}

__global__ void k_sx_xpos_clear(int64_t nx, const int32_t *xind, int64_t n, int32_t *xpos)
{
    const int64_t f = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (f >= nx) return;
    const int32_t c = xind[f];
    if (c >= 0 && c < n) xpos[c] = 0;
}

template <int SX>
__device__ __forceinline__ unsigned long long sx_key(int64_t x, int32_t c, int64_t f)
{
    if (SX == SX_SELECT2NDMIN) return ~((unsigned long long)x ^ kSign);
    if (SX == SX_SELECTMAX) return (unsigned long long)x ^ kSign;
    return ((unsigned long long)(uint32_t)c << 32) | (uint32_t)f;  // SX_SELECT2ND
}

// fn(f, p) for every entry p of the columns of the vector's entries f: blocks
// take kSxChunk entries at a time, whose products their threads share out (few
// enough that a vector of 2000 entries keeps 63 blocks busy, not 8).
constexpr int kSxChunk = 32;

template <class F>
__device__ __forceinline__ void sx_products(const int64_t *cp, const int32_t *xind, int64_t nx, int64_t n,
                                            unsigned long long *work, F &&fn)
{
    __shared__ int64_t s_seg[kSxChunk];
    __shared__ int64_t s_off[kSxChunk + 1];
    __shared__ int64_t s_base;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid < 32) {
            long long base = 0;
            if (tid == 0) base = (long long)atomicAdd(work, (unsigned long long)kSxChunk);
            base = __shfl_sync(0xffffffffu, base, 0);
            int64_t len = 0;
            if (base + tid < nx) {
                const int32_t c = xind[base + tid];
                if (c >= 0 && c < n) {
                    s_seg[tid] = cp[c];
                    len = cp[c + 1] - cp[c];
                }
            }
            int64_t x = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (tid >= o) x += y;
            }
            s_off[tid] = x - len;
            if (tid == 31) {
                s_off[32] = x;
                s_base = base;
            }
        }
        __syncthreads();
        const int64_t base = s_base, tot = s_off[kSxChunk];
        if (base >= nx) break;  // block-uniform
        for (int64_t j = tid; j < tot; j += kSxThreads) {
            int lo = 0;
#pragma unroll
            for (int step = kSxChunk / 2; step; step >>= 1)
                if (s_off[lo + step] <= j) lo += step;
            fn(base + lo, s_seg[lo] + (j - s_off[lo]));
        }
        __syncthreads();
    }
}

// Push: per product one atomicMax of the column's key into spa[r] (PlusTimes:
// a count, where `count` asks for it) and the touched mark.  A vector that
// k_sx_xpos found at fault brings nothing: distinct columns keep a row's count,
// and the total, within the matrix's entries (below 2^31), which the 32-bit
// places of the products rely on; a column named 2^16 times would pass them.
template <int SX>
__global__ void __launch_bounds__(kSxThreads) k_sx_expand(const int64_t *cp, const int32_t *row, const int32_t *xind,
                                                          const int64_t *xval, int64_t nx, int64_t n,
                                                          unsigned long long *spa, uint32_t *mark,
                                                          unsigned long long *work, const int32_t *err, bool count)
{
    if (*err != 0) return;
    sx_products(cp, xind, nx, n, work, [&](int64_t f, int64_t p) {
        const int32_t r = row[p];
        if (SX == SX_PLUSTIMES) {
            if (count) atomicAdd(&spa[r], 1ull);
        } else
            atomicMax(&spa[r], sx_key<SX>(xval[f], xind[f], f));
        const uint32_t bit = 1u << (r & 31);
        if (!(mark[r >> 5] & bit)) atomicOr(&mark[r >> 5], bit);
    });
}

__global__ void k_sx_counts(const uint32_t *mark, int64_t words, int64_t *cnt)
{
    const int64_t w = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w < words) cnt[w] = __popc(mark[w]);
}

// PlusTimes: touched rows (low 32 bits) and their products (high 32 bits).
__global__ void k_sx_counts_sum(const uint32_t *mark, int64_t words, const unsigned long long *spa, int64_t *cnt)
{
    const int64_t w = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= words) return;
    const uint32_t x = mark[w];
    unsigned long long c = 0;
    for (uint32_t bits = x; bits; bits &= bits - 1) c += spa[w * 32 + __ffs(bits) - 1];
    cnt[w] = (int64_t)((c << 32) | (unsigned)__popc(x));
}

// PlusTimes: touched rows in ascending order and the place of their products
// (off, and spa as a running cursor); clears the marks.
__global__ void k_sx_places(uint32_t *mark, int64_t words, const int64_t *pos, unsigned long long *spa, int32_t *yind,
                            uint32_t *off)
{
    const int64_t w = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= words) return;
    const unsigned long long at = (unsigned long long)pos[w];
    uint32_t p = (uint32_t)at, o = (uint32_t)(at >> 32);
    for (uint32_t bits = mark[w]; bits; bits &= bits - 1, ++p) {
        const int64_t r = w * 32 + __ffs(bits) - 1;
        const uint32_t c = (uint32_t)spa[r];
        yind[p] = (int32_t)r;
        off[p] = o;
        spa[r] = o;
        o += c;
    }
    mark[w] = 0;
    if (w == words - 1) off[p] = o;
}

// Touched rows in ascending order with their values (select semirings);
// clears the marks and keys.
template <int SX>
__global__ void k_sx_emit(uint32_t *mark, int64_t words, const int64_t *pos, unsigned long long *spa,
                          const int64_t *xval, int32_t *yind, int64_t *yval)
{
    const int64_t w = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (w >= words) return;
    uint32_t bits = mark[w];
    int64_t p = SX == SX_PLUSTIMES ? pos[w] & 0xffffffff : pos[w];
    while (bits) {
        const int b = __ffs(bits) - 1;
        bits &= bits - 1;
        const int64_t r = w * 32 + b;
        yind[p] = (int32_t)r;
        if (SX == SX_PLUSTIMES) {
            spa[r] = 0;
        } else {
            const unsigned long long k = spa[r];
            spa[r] = 0;
            int64_t v;
            if (SX == SX_SELECT2NDMIN)
                v = (int64_t)(~k ^ kSign);
            else if (SX == SX_SELECTMAX)
                v = (int64_t)(k ^ kSign);
            else
                v = xval[(uint32_t)(k & 0xffffffffu)];
            yval[p] = v;
        }
        ++p;
    }
    mark[w] = 0;
}

template <typename V>
__device__ __forceinline__ V sx_mul(V a, V b)
{
    if constexpr (std::is_same<V, double>::value) return __dmul_rn(a, b);
    else if constexpr (std::is_same<V, float>::value) return __fmul_rn(a, b);
    else return a * b;
}

template <typename V>
__device__ __forceinline__ V sx_add(V a, V b)
{
    if constexpr (std::is_same<V, double>::value) return __dadd_rn(a, b);
    else if constexpr (std::is_same<V, float>::value) return __fadd_rn(a, b);
    else return a + b;
}

constexpr int kSxThread = 8;      // products of a row folded by one thread
constexpr int kSxPullShare = 4;   // pull when the products times this exceed the matrix
// Matrices of fewer entries are always pulled: their longest row is a short
// chain, and the push has five launches more.  R-MAT, vectors of 30 / 2000 / 10000
// entries on the device, us pulled and pushed: 1.8*10^6 entries 84 161 295 and 91 197
// 344; 3.7*10^6 112 198 330 and 105 250 368; 7.6*10^6 141 204 348 and 115 201 311;
// 1.5*10^7 175 241 546 and 108 207 402; 3.1*10^7 237 343 662 and 114 193 310.
constexpr int64_t kSxPushNnz = 1 << 22;

// The row's products by one warp over its row-major entries, eight windows of
// 32 entries in flight; hits are folded left in ascending column order.
template <typename V>
__device__ __forceinline__ V sx_pull_row(int64_t b, int64_t e, const int32_t *col, const V *aval, const int32_t *xpos,
                                         const V *xval)
{
    constexpr int U = 8;
    const int lane = threadIdx.x & 31;
    V acc = V(0);
    bool have = false;
    for (int64_t base = b; base < e; base += 32 * U) {
        int32_t fx[U];
#pragma unroll
        for (int u = 0; u < U; ++u) fx[u] = base + u * 32 + lane < e ? col[base + u * 32 + lane] : -1;
#pragma unroll
        for (int u = 0; u < U; ++u) fx[u] = fx[u] >= 0 ? xpos[fx[u]] : 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            unsigned bal = __ballot_sync(0xffffffffu, fx[u] != 0);
            if (!bal) continue;
            V prod = V(0);
            if (fx[u]) prod = sx_mul<V>(aval[base + u * 32 + lane], xval[fx[u] - 1]);
            while (bal) {
                const int l = __ffs(bal) - 1;
                bal &= bal - 1;
                const V pv = __shfl_sync(0xffffffffu, prod, l);
                acc = have ? sx_add<V>(acc, pv) : pv;
                have = true;
            }
        }
    }
    return acc;
}

// PlusTimes pull: one warp per touched row.
template <typename V>
__global__ void __launch_bounds__(256) k_sx_pull(int64_t ny, const int32_t *yind, const int64_t *rowptr,
                                                 const int32_t *col, const V *aval, const int32_t *xpos,
                                                 const V *xval, V *yval)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t i = warp; i < ny; i += nwarps) {
        const int32_t r = yind[i];
        const V acc = sx_pull_row<V>(rowptr[r], rowptr[r + 1], col, aval, xpos, xval);
        if (lane == 0) yval[i] = acc;
    }
}

// PlusTimes push: the products of the vector's columns, each at the next place
// of its row (rows that will be pulled need none).
template <typename V>
__global__ void __launch_bounds__(kSxThreads) k_sx_scatter(const int64_t *cp, const int32_t *row, const V *aval,
                                                           const int32_t *xind, const V *xval, int64_t nx, int64_t n,
                                                           unsigned long long *spa, int32_t *pent, V *pval,
                                                           unsigned long long *work)
{
    sx_products(cp, xind, nx, n, work, [&](int64_t f, int64_t p) {
        const unsigned long long at = atomicAdd(&spa[row[p]], 1ull);
        pent[at] = (int32_t)p;
        pval[at] = sx_mul<V>(aval[p], xval[f]);
    });
}

// Every touched row folds its products in the order of their entries; the row's
// cursor goes back to zero.
template <typename V>
__global__ void __launch_bounds__(256) k_sx_fold(int64_t ny, const int32_t *yind, const uint32_t *off,
                                                 const int32_t *pent, const V *pval, unsigned long long *spa,
                                                 V *yval, int32_t *longs, unsigned long long *nlong)
{
    const int lane = threadIdx.x & 31;
    for (int64_t i0 = int64_t(blockIdx.x) * blockDim.x; i0 < ny; i0 += int64_t(gridDim.x) * blockDim.x) {
        const int64_t i = i0 + threadIdx.x;
        uint32_t o = 0, n = 0;
        if (i < ny) {
            o = off[i];
            n = off[i + 1] - o;
            spa[yind[i]] = 0;
            if (n <= kSxThread) {
                V acc = V(0);
                int32_t done = -1;  // the entries up to this one are folded
                for (uint32_t k = 0; k < n; ++k) {
                    int32_t next = INT32_MAX;
                    V v = V(0);
                    for (uint32_t q = 0; q < n; ++q) {
                        const int32_t c = pent[o + q];
                        if (c > done && c < next) {
                            next = c;
                            v = pval[o + q];
                        }
                    }
                    acc = k ? sx_add<V>(acc, v) : v;
                    done = next;
                }
                yval[i] = acc;
            }
        }
        unsigned more = __ballot_sync(0xffffffffu, n > kSxThread);
        while (more) {
            const int l = __ffs(more) - 1;
            more &= more - 1;
            const uint32_t ro = __shfl_sync(0xffffffffu, o, l), rn = __shfl_sync(0xffffffffu, n, l);
            const int64_t ri = i0 + (threadIdx.x & ~31) + l;
            if (rn > 32) {  // a block's work
                if (lane == 0) longs[atomicAdd(nlong, 1ull)] = (int32_t)ri;
                continue;
            }
            V acc = V(0);
            unsigned c = lane < (int)rn ? (unsigned)pent[ro + lane] : 0xffffffffu;
            const V v = lane < (int)rn ? pval[ro + lane] : V(0);
            for (uint32_t k = 0; k < rn; ++k) {
                const unsigned next = __reduce_min_sync(0xffffffffu, c);
                const int at = __ffs(__ballot_sync(0xffffffffu, c == next)) - 1;
                const V pv = __shfl_sync(0xffffffffu, v, at);
                acc = k ? sx_add<V>(acc, pv) : pv;
                if (lane == at) c = 0xffffffffu;
            }
            if (lane == 0) yval[ri] = acc;
        }
    }
}

// Rows of more than 32 products, a block each: the products are sorted by
// entry in shared memory (bitonic) and folded by one thread, the chain that
// the order asks for; rows of more than kSxSort are pulled.
constexpr int kSxSort = 2048;

template <typename V>
__global__ void __launch_bounds__(256) k_sx_fold_long(const int32_t *longs, const unsigned long long *nlong,
                                                      const int32_t *yind, const uint32_t *off, const int32_t *pent,
                                                      const V *pval, const int64_t *rowptr, const int32_t *col,
                                                      const V *aval, const int32_t *xpos, const V *xval, V *yval)
{
    __shared__ uint64_t key[kSxSort];
    __shared__ V val[kSxSort];
    const int tid = threadIdx.x;
    const int64_t count = (int64_t)*nlong;
    for (int64_t q = blockIdx.x; q < count; q += gridDim.x) {
        const int32_t i = longs[q];
        const uint32_t o = off[i];
        const int n = (int)(off[i + 1] - o);
        if (n > kSxSort) {
            if (tid < 32) {
                const int32_t r = yind[i];
                const V acc = sx_pull_row<V>(rowptr[r], rowptr[r + 1], col, aval, xpos, xval);
                if (tid == 0) yval[i] = acc;
            }
            continue;
        }
        int N = 64;
        while (N < n) N <<= 1;
        for (int k = tid; k < N; k += 256)
            key[k] = k < n ? ((uint64_t)(uint32_t)pent[o + k] << 32) | (uint32_t)k : ~0ull;
        __syncthreads();
        for (int k2 = 2; k2 <= N; k2 <<= 1) {
            for (int j = k2 >> 1; j > 0; j >>= 1) {
                for (int u = tid; u < (N >> 1); u += 256) {
                    const int lo = ((u & ~(j - 1)) << 1) | (u & (j - 1)), hi = lo + j;
                    const uint64_t x0 = key[lo], x1 = key[hi];
                    if ((x0 > x1) == ((lo & k2) == 0)) {
                        key[lo] = x1;
                        key[hi] = x0;
                    }
                }
                __syncthreads();
            }
        }
        for (int k = tid; k < n; k += 256) val[k] = pval[o + (uint32_t)key[k]];
        __syncthreads();
        if (tid == 0) {
            V acc = val[0];
#pragma unroll 8
            for (int k = 1; k < n; ++k) acc = sx_add<V>(acc, val[k]);
            yval[i] = acc;
        }
        __syncthreads();
    }
}

static void plan_release(SpmspvPlan *p)
{
    if (!p->ctx) return;
    cudaSetDevice(p->ctx->device);
    cudaStreamSynchronize(p->ctx->stream);
    if (p->have_rm) spmv_plan_release(&p->rm);
    device_free(p->ctx, p->cp);
    device_free(p->ctx, p->row);
    device_free(p->ctx, p->cval);
    device_free(p->ctx, p->spa);
    device_free(p->ctx, p->mark);
    device_free(p->ctx, p->pos);
    device_free(p->ctx, p->xpos);
    device_free(p->ctx, p->err);
    device_free(p->ctx, p->work);
    cudaStreamSynchronize(p->ctx->stream);
}

static int plan_build(SpmspvPlan *p, const gbc_matrix *Am)
{
    Context *ctx = p->ctx;
    cudaStream_t s = ctx->stream;
    Workspace ws(ctx);
    DevMatrix A;
    GBC_TRY(upload(ws, Am, p->vt, &A));
    p->m = A.nrow;
    p->n = A.ncol;
    p->nnz = A.nnz;
    if (A.nrow >= (int64_t(1) << 31) || A.ncol >= (int64_t(1) << 31))
        return fail(GBC_EOVERFLOW, "SpMSpV plan: dimensions must be below 2^31");
    p->words = (p->m + 31) / 32;
    int64_t *cnt = nullptr;
    GBC_TRY(ws.alloc_n(&cnt, p->n + 1));
    GBC_TRY(device_alloc(ctx, (void **)&p->cp, (p->n + 1) * sizeof(int64_t)));
    GBC_TRY(device_alloc(ctx, (void **)&p->row, (p->nnz + 1) * sizeof(int32_t)));
    GBC_TRY(device_alloc(ctx, (void **)&p->spa, (p->m + 1) * sizeof(unsigned long long)));
    GBC_TRY(device_alloc(ctx, (void **)&p->mark, (p->words + 1) * sizeof(uint32_t)));
    GBC_TRY(device_alloc(ctx, (void **)&p->pos, (p->words + 1) * sizeof(int64_t)));
    GBC_TRY(device_alloc(ctx, (void **)&p->xpos, (p->n + 1) * sizeof(int32_t)));
    GBC_TRY(device_alloc(ctx, (void **)&p->err, sizeof(int32_t)));
    GBC_TRY(device_alloc(ctx, (void **)&p->work, sizeof(unsigned long long)));
    GBC_CUDA_TRY(cudaMemsetAsync(cnt, 0, (p->n + 1) * sizeof(int64_t), s));
    GBC_CUDA_TRY(cudaMemsetAsync(p->spa, 0, (p->m + 1) * sizeof(unsigned long long), s));
    GBC_CUDA_TRY(cudaMemsetAsync(p->mark, 0, (p->words + 1) * sizeof(uint32_t), s));
    GBC_CUDA_TRY(cudaMemsetAsync(p->xpos, 0, (p->n + 1) * sizeof(int32_t), s));
    GBC_CUDA_TRY(cudaMemsetAsync(p->err, 0, sizeof(int32_t), s));
    if (A.nzc > 0) {
        const int grid = (int)std::min<int64_t>((A.nzc + 7) / 8, (int64_t)ctx->num_sms * 16);
        k_sx_prep<<<grid, 256, 0, s>>>(A.nzc, p->m, p->n, p->nnz, A.cp, A.jc, A.ir, cnt, p->row, p->err);
        note_launch();
    }
    GBC_TRY(exclusive_scan_i64(ws, cnt, p->cp, p->n, s));
    int32_t herr = 0;
    GBC_CUDA_TRY(cudaMemcpyAsync(&herr, p->err, sizeof(herr), cudaMemcpyDeviceToHost, s));
    GBC_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr & 1) return fail(GBC_EINVAL, "SpMSpV plan: malformed column pointers or column ids");
    if (herr & 2) return fail(GBC_EINVAL, "SpMSpV plan: row id out of range");
    if (p->vt == GBC_F64 || p->vt == GBC_F32 || p->vt == GBC_I64) {
        const size_t vs = value_size(p->vt);
        GBC_TRY(device_alloc(ctx, &p->cval, (p->nnz + 1) * vs));
        if (A.num) {
            GBC_CUDA_TRY(cudaMemcpyAsync(p->cval, A.num, p->nnz * vs, cudaMemcpyDeviceToDevice, s));
        } else if (p->nnz > 0) {
            const unsigned g = (unsigned)((p->nnz + 255) / 256);
            if (p->vt == GBC_F64) k_sx_ones<double><<<g, 256, 0, s>>>(p->nnz, static_cast<double *>(p->cval));
            if (p->vt == GBC_F32) k_sx_ones<float><<<g, 256, 0, s>>>(p->nnz, static_cast<float *>(p->cval));
            if (p->vt == GBC_I64) k_sx_ones<int64_t><<<g, 256, 0, s>>>(p->nnz, static_cast<int64_t *>(p->cval));
            note_launch();
        }
        p->rm.ctx = ctx;
        p->rm.vt = p->vt;
        p->rm.tiles = false;
        p->have_rm = true;
        GBC_TRY(spmv_plan_build(&p->rm, Am));
    }
    return GBC_OK;
}

// A call that ends early, by a failed allocation or launch, clears the plan's
// scratch on its way out; `done` says that its kernels have.
struct SxRestore {
    SpmspvPlan *p;
    cudaStream_t s;
    bool done = false;
    ~SxRestore()
    {
        if (done) return;
        cudaMemsetAsync(p->spa, 0, (p->m + 1) * sizeof(unsigned long long), s);
        cudaMemsetAsync(p->mark, 0, (p->words + 1) * sizeof(uint32_t), s);
        cudaMemsetAsync(p->xpos, 0, (p->n + 1) * sizeof(int32_t), s);
    }
};

// The pushed products' arrays.
template <typename V>
struct SxProducts {
    uint32_t *off = nullptr;   // [ny + 1] where every touched row's products begin
    int32_t *pent = nullptr;   // [nprod] their entries
    V *pval = nullptr;         // [nprod]
    int32_t *longs = nullptr;  // rows of more than 32 products
    unsigned long long *nlong = nullptr;
    int reserve(Workspace &ws, int64_t ny, int64_t nprod)
    {
        GBC_TRY(ws.alloc_n(&off, ny + 1));
        GBC_TRY(ws.alloc_n(&pent, nprod));
        GBC_TRY(ws.alloc_n(&pval, nprod));
        GBC_TRY(ws.alloc_n(&longs, nprod / 33 + 1));
        return ws.alloc_n(&nlong, 1);
    }
};

template <int SX, typename V>
static int sx_run(SpmspvPlan *p, Workspace &ws, const int32_t *dx, const void *dv, int64_t nx, int32_t **yi,
                  void **yv, int64_t *ny, bool host_out)
{
    Context *ctx = p->ctx;
    cudaStream_t s = ctx->stream;
    const bool push = SX == SX_PLUSTIMES && p->nnz >= kSxPushNnz;
    GBC_CUDA_TRY(cudaMemsetAsync(p->err, 0, sizeof(int32_t), s));
    GBC_CUDA_TRY(cudaMemsetAsync(p->work, 0, sizeof(unsigned long long), s));
    SxRestore restore{p, s};
    if (nx > 0) {
        k_sx_xpos<<<(unsigned)((nx + 255) / 256), 256, 0, s>>>(nx, dx, p->n, p->xpos, p->err);
        const int grid = (int)std::min<int64_t>((int64_t)ctx->num_sms * 8, (nx + kSxChunk - 1) / kSxChunk);
        k_sx_expand<SX><<<grid, kSxThreads, 0, s>>>(p->cp, p->row, dx, static_cast<const int64_t *>(dv), nx, p->n,
                                                    p->spa, p->mark, p->work, p->err, push);
        note_launches(2);
    }
    int64_t *cnt = nullptr;
    GBC_TRY(ws.alloc_n(&cnt, p->words + 1));
    if (p->words > 0) {
        if (push)
            k_sx_counts_sum<<<(unsigned)((p->words + 255) / 256), 256, 0, s>>>(p->mark, p->words, p->spa, cnt);
        else
            k_sx_counts<<<(unsigned)((p->words + 255) / 256), 256, 0, s>>>(p->mark, p->words, cnt);
        note_launch();
    }
    GBC_TRY(exclusive_scan_i64(ws, cnt, p->pos, p->words, s));
    GBC_TRY(read_i64(ctx, p->pos + p->words, ny));
    const int64_t nprod = push ? (int64_t)((uint64_t)*ny >> 32) : 0;
    if (push) *ny &= 0xffffffff;
    if (host_out) {
        GBC_TRY(ws.alloc_n(yi, *ny + 1));
        void *b = nullptr;
        GBC_TRY(ws.alloc(&b, (*ny + 1) * sizeof(V)));
        *yv = b;
    }
    SxProducts<V> q;  // (without room for them the rows are pulled)
    if (push && *ny > 0 && nprod * kSxPullShare <= p->nnz && q.reserve(ws, *ny, nprod) == GBC_OK) {
        GBC_CUDA_TRY(cudaMemsetAsync(q.nlong, 0, sizeof(unsigned long long), s));
        k_sx_places<<<(unsigned)((p->words + 255) / 256), 256, 0, s>>>(p->mark, p->words, p->pos, p->spa, *yi, q.off);
        GBC_CUDA_TRY(cudaMemsetAsync(p->work, 0, sizeof(unsigned long long), s));
        const int grid = (int)std::min<int64_t>((int64_t)ctx->num_sms * 8, (nx + kSxChunk - 1) / kSxChunk);
        k_sx_scatter<V><<<grid, kSxThreads, 0, s>>>(p->cp, p->row, static_cast<const V *>(p->cval), dx,
                                                    static_cast<const V *>(dv), nx, p->n, p->spa, q.pent, q.pval, p->work);
        k_sx_fold<V><<<(int)std::min<int64_t>((*ny + 255) / 256, (int64_t)ctx->num_sms * 8), 256, 0, s>>>(
            *ny, *yi, q.off, q.pent, q.pval, p->spa, static_cast<V *>(*yv), q.longs, q.nlong);
        k_sx_fold_long<V><<<(int)std::min<int64_t>(nprod / 33 + 1, (int64_t)ctx->num_sms * 6), 256, 0, s>>>(
            q.longs, q.nlong, *yi, q.off, q.pent, q.pval, p->rm.rowptr, p->rm.col, static_cast<const V *>(p->rm.val),
            p->xpos, static_cast<const V *>(dv), static_cast<V *>(*yv));
        note_launches(4);
    } else {
        if (p->words > 0) {
            k_sx_emit<SX><<<(unsigned)((p->words + 255) / 256), 256, 0, s>>>(
                p->mark, p->words, p->pos, p->spa, static_cast<const int64_t *>(dv), *yi,
                SX == SX_PLUSTIMES ? nullptr : static_cast<int64_t *>(*yv));
            note_launch();
        }
        if (SX == SX_PLUSTIMES && *ny > 0) {
            const int grid = (int)std::min<int64_t>((*ny + 7) / 8, (int64_t)ctx->num_sms * 16);
            k_sx_pull<V><<<grid, 256, 0, s>>>(*ny, *yi, p->rm.rowptr, p->rm.col, static_cast<const V *>(p->rm.val),
                                              p->xpos, static_cast<const V *>(dv), static_cast<V *>(*yv));
            note_launch();
        }
    }
    if (nx > 0) {
        k_sx_xpos_clear<<<(unsigned)((nx + 255) / 256), 256, 0, s>>>(nx, dx, p->n, p->xpos);
        note_launch();
    }
    GBC_CUDA_TRY(cudaGetLastError());
    restore.done = true;
    int32_t herr = 0;
    GBC_CUDA_TRY(cudaMemcpyAsync(&herr, p->err, sizeof(herr), cudaMemcpyDeviceToHost, s));
    GBC_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr & 1) return fail(GBC_EINVAL, "vector index out of range");
    if (herr & 2) return fail(GBC_EINVAL, "repeated vector index");
    return GBC_OK;
}

}  // namespace gbc

using namespace gbc;

struct gbc_spmspv_plan : gbc::SpmspvPlan {};

extern "C" {

int gbc_spmspv_plan_create(gbc_context *ctx, int vt, const gbc_matrix *A, gbc_spmspv_plan **out)
{
    if (!ctx || !A || !out) return fail(GBC_EINVAL, "null argument");
    *out = nullptr;
    if (vt != GBC_F64 && vt != GBC_F32 && vt != GBC_I64 && vt != GBC_BOOL) return fail(GBC_EINVAL, "bad value type");
    GBC_CUDA_TRY(cudaSetDevice(ctx->device));
    gbc_spmspv_plan *p = new gbc_spmspv_plan();
    p->ctx = ctx;
    p->vt = vt;
    const int rc = plan_build(p, A);
    if (rc != GBC_OK) {
        gbc_spmspv_plan_destroy(p);
        return rc;
    }
    *out = p;
    return GBC_OK;
}

int gbc_spmspv_plan_destroy(gbc_spmspv_plan *p)
{
    if (!p) return GBC_OK;
    plan_release(p);
    delete p;
    return GBC_OK;
}

int gbc_spmspv(gbc_context *ctx, gbc_spmspv_plan *p, int sr, const int32_t *indx, const void *numx, int32_t veclen,
               int32_t *indy, void *numy, int32_t *nnzy, int where)
{
    if (!ctx || !p || !nnzy) return fail(GBC_EINVAL, "null argument");
    if (veclen < 0) return fail(GBC_EINVAL, "negative vector length");
    if (veclen > 0 && (!indx || !numx)) return fail(GBC_EINVAL, "null vector");
    if (where != GBC_HOST && where != GBC_DEVICE) return fail(GBC_EINVAL, "bad memory location");
    int sx = -1;
    size_t xs = 8;
    switch (sr) {
        case GBC_SR_SELECT2NDMIN: sx = SX_SELECT2NDMIN; break;
        case GBC_SR_SELECT2ND: sx = SX_SELECT2ND; break;
        case GBC_SR_SELECTMAX: sx = SX_SELECTMAX; break;
        case GBC_SR_PLUSTIMES:
            if (p->vt == GBC_BOOL) return fail(GBC_EUNSUPPORTED, "PlusTimes SpMSpV needs a numeric matrix");
            sx = SX_PLUSTIMES;
            xs = value_size(p->vt);
            break;
        default: return fail(GBC_EUNSUPPORTED, "semiring not instantiated for SpMSpV");
    }
    GBC_CUDA_TRY(cudaSetDevice(ctx->device));
    p->ctx = ctx;
    p->rm.ctx = ctx;
    cudaStream_t s = ctx->stream;
    Workspace ws(ctx);
    const int32_t *dx = indx;
    const void *dv = numx;
    if (where == GBC_HOST && veclen > 0) {
        int32_t *a = nullptr;
        void *b = nullptr;
        GBC_TRY(ws.alloc_n(&a, veclen));
        GBC_TRY(ws.alloc(&b, veclen * xs));
        GBC_CUDA_TRY(cudaMemcpyAsync(a, indx, veclen * sizeof(int32_t), cudaMemcpyHostToDevice, s));
        GBC_CUDA_TRY(cudaMemcpyAsync(b, numx, veclen * xs, cudaMemcpyHostToDevice, s));
        dx = a;
        dv = b;
    }
    int32_t *yi = indy;
    void *yv = numy;
    int64_t ny = 0;
    const bool host_out = where == GBC_HOST;
    int rc;
    switch (sx) {
        case SX_SELECT2NDMIN: rc = sx_run<SX_SELECT2NDMIN, int64_t>(p, ws, dx, dv, veclen, &yi, &yv, &ny, host_out); break;
        case SX_SELECT2ND: rc = sx_run<SX_SELECT2ND, int64_t>(p, ws, dx, dv, veclen, &yi, &yv, &ny, host_out); break;
        case SX_SELECTMAX: rc = sx_run<SX_SELECTMAX, int64_t>(p, ws, dx, dv, veclen, &yi, &yv, &ny, host_out); break;
        default:
            if (p->vt == GBC_F64)
                rc = sx_run<SX_PLUSTIMES, double>(p, ws, dx, dv, veclen, &yi, &yv, &ny, host_out);
            else if (p->vt == GBC_F32)
                rc = sx_run<SX_PLUSTIMES, float>(p, ws, dx, dv, veclen, &yi, &yv, &ny, host_out);
            else
                rc = sx_run<SX_PLUSTIMES, int64_t>(p, ws, dx, dv, veclen, &yi, &yv, &ny, host_out);
    }
    if (rc != GBC_OK) return rc;
    const size_t ys = sx == SX_PLUSTIMES ? xs : 8;
    if (host_out && ny > 0) {
        GBC_CUDA_TRY(cudaMemcpyAsync(indy, yi, ny * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        GBC_CUDA_TRY(cudaMemcpyAsync(numy, yv, ny * ys, cudaMemcpyDeviceToHost, s));
        GBC_CUDA_TRY(cudaStreamSynchronize(s));
    }
    *nnzy = (int32_t)ny;
    return GBC_OK;
}

int gbc_spmspv_plan_info(const gbc_spmspv_plan *p, int64_t *nrow, int64_t *ncol, int64_t *nnz)
{
    if (!p) return fail(GBC_EINVAL, "null argument");
    if (nrow) *nrow = p->m;
    if (ncol) *ncol = p->n;
    if (nnz) *nnz = p->nnz;
    return GBC_OK;
}

}  // extern "C"
