// Sparse matrix x dense vector over a semiring, y <- y (+) A x: the local
// multiply of dcsc_gespmv / dcsc_gespmv_threaded (Friends.h:63-175), whose
// per-row update is SR::axpy(a, x[col], y[row]) over A's columns in order.
//
// GPU form: a plan holds A row-major (rows ascending, each row's entries in
// ascending column order) built once on the device by a stable LSD radix
// sort of the column-major entries by row.  A thread takes kSpmvPer consecutive
// entries whatever rows they belong to: it folds them in order, whole rows are
// done there, and the open sums at its ends are joined by a segmented scan over
// the block and, for rows that cross blocks, by a second small kernel.
// The order is fixed, so repeated runs are bit-identical; for min-type,
// boolean and integer semirings every order gives the reference's result
// exactly, and for PlusTimes on floating values the sum differs from the
// reference's column-order sum only by rounding.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "gbc_internal.cuh"
#include "semiring.cuh"
#include "spmv_plan.cuh"

namespace gbc {

constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
constexpr int kRsRounds = 8;
constexpr int kRsTile = kRsThreads * kRsRounds;  // items per block and pass
constexpr int kRsRadix = 256;

// per-entry column ids of a CSC/DCSC
__global__ void k_entry_cols(int64_t nzc, const int64_t *cp, const int64_t *jc, int32_t *col)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    for (int64_t i = warp; i < nzc; i += nwarps) {
        const int32_t c = (int32_t)(jc ? jc[i] : i);
        for (int64_t p = cp[i] + lane; p < cp[i + 1]; p += 32) col[p] = c;
    }
}

__global__ void k_row_keys(int64_t n, const int64_t *ir, int64_t m, uint32_t *key, int32_t *idx, int64_t *rowcnt,
                           int32_t *err)
{
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int64_t r = ir[i];
    if (r < 0 || r >= m) {
        atomicOr(err, 1);
        r = 0;
    }
    key[i] = (uint32_t)r;
    idx[i] = (int32_t)i;
    atomicAdd((unsigned long long *)&rowcnt[r], 1ull);
}

// Digit counts of one tile of kRsTile items.
__global__ void __launch_bounds__(kRsThreads) k_rs_count(const uint32_t *key, int64_t n, int shift, int64_t *hist)
{
    __shared__ int cnt[kRsRadix];
    cnt[threadIdx.x] = 0;
    __syncthreads();
    const int64_t t0 = int64_t(blockIdx.x) * kRsTile;
    for (int i = threadIdx.x; i < kRsTile; i += kRsThreads) {
        const int64_t it = t0 + i;
        if (it < n) atomicAdd(&cnt[(key[it] >> shift) & (kRsRadix - 1)], 1);
    }
    __syncthreads();
    hist[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = cnt[threadIdx.x];
}

// Stable scatter of one tile: items keep their order within a digit.
// off[d * nblocks + b] is the first output slot of digit d for tile b.
__global__ void __launch_bounds__(kRsThreads) k_rs_scatter(const uint32_t *key_in, const int32_t *val_in, int64_t n,
                                                           int shift, const int64_t *off, uint32_t *key_out,
                                                           int32_t *val_out)
{
    __shared__ int64_t base[kRsWarps][kRsRadix];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1;
    for (int d = threadIdx.x; d < kRsWarps * kRsRadix; d += kRsThreads) base[d / kRsRadix][d % kRsRadix] = 0;
    __syncthreads();
    // warp w owns items [t0 + w*256, t0 + (w+1)*256) in 8 rounds of 32
    const int64_t w0 = int64_t(blockIdx.x) * kRsTile + (int64_t)w * (kRsTile / kRsWarps);
    for (int r = 0; r < kRsRounds; ++r) {
        const int64_t it = w0 + r * 32 + lane;
        if (it < n) atomicAdd((unsigned long long *)&base[w][(key_in[it] >> shift) & (kRsRadix - 1)], 1ull);
    }
    __syncthreads();
    {
        const int d = threadIdx.x;  // kRsThreads == kRsRadix
        int64_t run = off[(int64_t)d * gridDim.x + blockIdx.x];
        for (int u = 0; u < kRsWarps; ++u) {
            const int64_t c = base[u][d];
            base[u][d] = run;
            run += c;
        }
    }
    __syncthreads();
    for (int r = 0; r < kRsRounds; ++r) {
        const int64_t it = w0 + r * 32 + lane;
        const bool act = it < n;
        const uint32_t k = act ? key_in[it] : 0;
        const int d = act ? (int)((k >> shift) & (kRsRadix - 1)) : 0;
        // lanes holding the same digit, from eight ballots
        unsigned peers = __ballot_sync(0xffffffffu, act);
#pragma unroll
        for (int bit = 0; bit < 8; ++bit) {
            const unsigned bb = __ballot_sync(0xffffffffu, act && ((d >> bit) & 1));
            peers &= ((d >> bit) & 1) ? bb : ~bb;
        }
        if (act) {
            const int64_t dst = base[w][d] + __popc(peers & lt);
            key_out[dst] = k;
            val_out[dst] = val_in[it];
        }
        __syncwarp();
        if (act && (peers & lt) == 0) base[w][d] += __popc(peers);
        __syncwarp();
    }
}

constexpr int kSpmvPer = 8;
constexpr int kSpmvThreads = 128;
constexpr int kSpmvTile = kSpmvPer * kSpmvThreads;

template <typename V>
__global__ void k_gather_rowmajor(int64_t n, const int32_t *perm, const int32_t *col_cm, const V *val_cm, V one,
                                  int32_t *col, V *val)
{
    const int64_t p = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const int32_t e = perm[p];
    col[p] = col_cm[e];
    val[p] = val_cm ? val_cm[e] : one;
}

// Rows with entries, their starts, and the row of every group of kSpmvPer entries.
__global__ void k_spmv_has(int64_t m, const int64_t *rowptr, int64_t *has)
{
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r < m) has[r] = rowptr[r + 1] > rowptr[r];
}

// A long row's groups are written by its whole warp: by one thread they took
// 1.3 ms of a plan with a row of 4*10^6 entries.
__global__ void k_spmv_mark(int64_t m, const int64_t *rowptr, const int64_t *index, int32_t *rows, uint32_t *starts,
                            int32_t *group_row)
{
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    int64_t s = 0, e = 0;
    int32_t i = 0;
    if (r < m) {
        s = rowptr[r];
        e = rowptr[r + 1];
    }
    if (e > s) {
        i = (int32_t)index[r];
        rows[i] = (int32_t)r;
        atomicOr(&starts[s >> 5], 1u << (s & 31));
    }
    const bool is_long = e - s > 32 * kSpmvPer;
    if (!is_long)
        for (int64_t g = (s + kSpmvPer - 1) / kSpmvPer; g * kSpmvPer < e; ++g) group_row[g] = i;
    for (unsigned todo = __ballot_sync(0xffffffffu, is_long); todo; todo &= todo - 1) {
        const int l = __ffs(todo) - 1;
        const int64_t ls = __shfl_sync(0xffffffffu, s, l), le = __shfl_sync(0xffffffffu, e, l);
        const int32_t li = __shfl_sync(0xffffffffu, i, l);
        for (int64_t g = (ls + kSpmvPer - 1) / kSpmvPer + lane; g * kSpmvPer < le; g += 32) group_row[g] = li;
    }
}

// acc + a * x.  Floating sums use a fused multiply-add: one rounding less, and
// half the fp64 instructions, which bound this kernel otherwise (GB300 issues
// two fp64 operations per SM and clock).
template <class SR>
__device__ __forceinline__ typename SR::V spmv_axpy(typename SR::V a, typename SR::V x, typename SR::V acc)
{
    typedef typename SR::V V;
    if constexpr (std::is_same<SR, PlusTimes<double>>::value)
        return __fma_rn(a, x, acc);
    else if constexpr (std::is_same<SR, PlusTimes<float>>::value)
        return __fmaf_rn(a, x, acc);
    else
        return SR::add(acc, (V)SR::mul(a, x));
}

// One tile of kSpmvTile entries.  Bound by the latency of the gathers of x (an
// L2 sector per entry) behind the entries' own loads, and by the fp64 pipe.
// R-MAT scale 20 fp64, 31 M entries, 386 us by rows (eight lanes or a warp per
// row and a shuffle tree for each): 182 us with 8 entries a thread and 128
// threads (64: 189, 256: 214, 512: 276); with 256 threads 205 to 214 us, 263
// with 16 entries a thread, 255 with 4, 331 with the gathers in entry order and
// handed over through shared memory.
template <class SR>
__global__ void __launch_bounds__(kSpmvThreads) k_spmv_tiles(int64_t nnz, const uint32_t *starts,
                                                             const int32_t *group_row, const int32_t *rows,
                                                             const int32_t *col, const typename SR::V *val,
                                                             const typename SR::V *x, typename SR::V *y,
                                                             typename SR::V *edge, int32_t *edge_row)
{
    typedef typename SR::V V;
    constexpr int NW = kSpmvThreads / 32;
    __shared__ V s_row[kSpmvTile + 1];  // whole rows' sums, from the tile's first start on
    __shared__ V s_sum[NW];
    __shared__ int s_flag[NW], s_n[NW], s_r0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t group = int64_t(blockIdx.x) * kSpmvThreads + tid, base = group * kSpmvPer;
    const int count = (int)max((int64_t)0, min((int64_t)kSpmvPer, nnz - base));
    unsigned flags = 0;
    int cur = 0;  // the row that is open (index into rows); before the first entry: the row before it
    if (count > 0) {
        flags = (starts[base >> 5] >> (base & 31)) & ((1u << kSpmvPer) - 1);
        cur = group_row[group] - (int)(flags & 1);
    }
    V v[kSpmvPer];
    V xq[kSpmvPer];
    {
        int32_t c[kSpmvPer];
        if (count == kSpmvPer) {
#pragma unroll
            for (int k = 0; k < kSpmvPer; k += 4) {
                const int4 q = *reinterpret_cast<const int4 *>(col + base + k);
                memcpy(&c[k], &q, 16);
            }
            if constexpr (sizeof(V) >= 4) {
                constexpr int K = 16 / sizeof(V);
#pragma unroll
                for (int k = 0; k < kSpmvPer; k += K) {
                    const int4 q = *reinterpret_cast<const int4 *>(val + base + k);
                    memcpy(&v[k], &q, 16);
                }
            } else {
#pragma unroll
                for (int k = 0; k < kSpmvPer; ++k) v[k] = val[base + k];
            }
        } else {
#pragma unroll
            for (int k = 0; k < kSpmvPer; ++k) {
                c[k] = k < count ? col[base + k] : -1;
                v[k] = k < count ? val[base + k] : SR::one();
            }
        }
#pragma unroll
        for (int k = 0; k < kSpmvPer; ++k) xq[k] = c[k] >= 0 ? x[c[k]] : SR::one();
    }
    if (tid == 0) s_r0 = cur;
    // rows open before the tile and flags before each thread
    const int nf = __popc(flags);
    int before = nf;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += u;
    }
    if (lane == 31) s_n[warp] = before;
    before -= nf;
    __syncthreads();
    int total = 0;
#pragma unroll
    for (int u = 0; u < NW; ++u) {
        before += u < warp ? s_n[u] : 0;
        total += s_n[u];
    }
    // fold in order: head, the sum up to the thread's first start; whole rows; acc, the open sum at its end
    V acc = SR::zero(), head = SR::zero();
    bool seen = false;
    int at = before;  // starts before the next one: row at of the tile is open
#pragma unroll
    for (int k = 0; k < kSpmvPer; ++k) {
        if ((flags >> k) & 1) {
            if (seen)
                s_row[at] = acc;
            else
                head = acc;
            seen = true;
            ++at;
            acc = SR::zero();
        }
        if (k < count) acc = spmv_axpy<SR>(v[k], xq[k], acc);
    }
    // segmented inclusive scan of the open sums
    V sum = acc;
    bool flag = seen;
    if (!__all_sync(0xffffffffu, seen)) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const V su = __shfl_up_sync(0xffffffffu, sum, o);
            const bool fu = __shfl_up_sync(0xffffffffu, (int)flag, o) != 0;
            if (lane >= o && !flag) {
                sum = SR::add(su, sum);
                flag = fu;
            }
        }
    }
    if (lane == 31) {
        s_sum[warp] = sum;
        s_flag[warp] = flag;
    }
    V left = __shfl_up_sync(0xffffffffu, sum, 1);
    const bool left_flag = __shfl_up_sync(0xffffffffu, (int)flag, 1) != 0 && lane > 0;
    __syncthreads();
    V carry = SR::zero();
    for (int u = 0; u < warp; ++u) carry = s_flag[u] ? s_sum[u] : SR::add(carry, s_sum[u]);
    if (lane == 0)
        left = carry;
    else if (!left_flag)
        left = SR::add(carry, left);
    if (seen) s_row[before] = SR::add(left, head);  // the row that ends at the thread's first start
    if (tid == kSpmvThreads - 1) {
        edge[2 * (int64_t)blockIdx.x + 1] = flag ? sum : SR::add(carry, sum);
        if (total == 0) edge_row[blockIdx.x] = -2;
    }
    __syncthreads();
    if (tid == 0 && total > 0) {  // row 0 of the tile began before it
        edge[2 * (int64_t)blockIdx.x] = s_row[0];
        edge_row[blockIdx.x] = s_r0;
    }
    for (int k = 1 + tid; k < total; k += kSpmvThreads) {
        const int32_t r = rows[s_r0 + k];
        y[r] = SR::add(y[r], s_row[k]);
    }
}

// Rows that cross tiles: the open sum behind the last start of an earlier tile,
// the tiles without a start in between, and what the row has in tile b.  The
// last row ends behind the last tile (b == ntiles).
template <class SR>
__global__ void k_spmv_edges(int64_t ntiles, int64_t nrows, const int32_t *rows, const typename SR::V *edge,
                             const int32_t *edge_row, typename SR::V *y)
{
    typedef typename SR::V V;
    const int64_t b = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (b > ntiles) return;
    const int64_t i = b < ntiles ? edge_row[b] : nrows - 1;
    if (i < 0) return;
    int64_t u = b - 1;
    while (edge_row[u] == -2) --u;  // the first tile has a start
    V sum = edge[2 * u + 1];
    for (++u; u < b; ++u) sum = SR::add(sum, edge[2 * u + 1]);
    if (b < ntiles) sum = SR::add(sum, edge[2 * b]);
    const int32_t r = rows[i];
    y[r] = SR::add(y[r], sum);
}

template <typename V>
static int plan_values(SpmvPlan *p, Workspace &ws, const DevMatrix &A, const int32_t *perm, const int32_t *col_cm)
{
    GBC_TRY(device_alloc(p->ctx, &p->val, (p->nnz + 1) * sizeof(V)));
    if (p->nnz > 0) {
        k_gather_rowmajor<V><<<(unsigned)((p->nnz + 255) / 256), 256, 0, p->ctx->stream>>>(
            p->nnz, perm, col_cm, static_cast<const V *>(A.num), (V)1, p->col, static_cast<V *>(p->val));
        note_launch();
    }
    return GBC_OK;
}

int spmv_plan_build(SpmvPlan *p, const gbc_matrix *Am)
{
    Context *ctx = p->ctx;
    cudaStream_t s = ctx->stream;
    Workspace ws(ctx);
    DevMatrix A;
    GBC_TRY(upload(ws, Am, p->vt, &A));
    p->m = A.nrow;
    p->n = A.ncol;
    p->nnz = A.nnz;
    if (A.nnz >= (int64_t(1) << 31) || A.ncol >= (int64_t(1) << 31) || A.nrow >= (int64_t(1) << 32))
        return fail(GBC_EOVERFLOW, "SpMV plan: nnz and columns must be below 2^31, rows below 2^32");
    const int64_t n = A.nnz;
    int32_t *err = nullptr, *col_cm = nullptr, *idx[2] = {nullptr, nullptr};
    uint32_t *key[2] = {nullptr, nullptr};
    int64_t *rowcnt = nullptr;
    GBC_TRY(ws.alloc_n(&err, 4));
    GBC_CUDA_TRY(cudaMemsetAsync(err, 0, 4 * sizeof(int32_t), s));
    GBC_TRY(ws.alloc_n(&col_cm, n + 1));
    GBC_TRY(ws.alloc_n(&key[0], n + 1));
    GBC_TRY(ws.alloc_n(&key[1], n + 1));
    GBC_TRY(ws.alloc_n(&idx[0], n + 1));
    GBC_TRY(ws.alloc_n(&idx[1], n + 1));
    GBC_TRY(ws.alloc_n(&rowcnt, p->m + 1));
    GBC_CUDA_TRY(cudaMemsetAsync(rowcnt, 0, (p->m + 1) * sizeof(int64_t), s));
    GBC_TRY(device_alloc(ctx, (void **)&p->rowptr, (p->m + 1) * sizeof(int64_t)));
    GBC_TRY(device_alloc(ctx, (void **)&p->col, (n + 1) * sizeof(int32_t)));
    if (A.nzc > 0) {
        k_entry_cols<<<(unsigned)std::min<int64_t>((A.nzc + 7) / 8, (int64_t)ctx->num_sms * 16), 256, 0, s>>>(
            A.nzc, A.cp, A.jc, col_cm);
        note_launch();
    }
    if (n > 0) {
        k_row_keys<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, A.ir, p->m, key[0], idx[0], rowcnt, err);
        note_launch();
    }
    GBC_TRY(exclusive_scan_i64(ws, rowcnt, p->rowptr, p->m, s));
    // stable LSD radix sort of the entries by row (8-bit digits)
    int cur = 0;
    if (n > 0) {
        int bits = 0;
        while (bits < 32 && (uint64_t(1) << bits) < (uint64_t)p->m) ++bits;
        const int64_t nblocks = (n + kRsTile - 1) / kRsTile;
        int64_t *hist = nullptr;
        GBC_TRY(ws.alloc_n(&hist, (size_t)kRsRadix * nblocks + 1));
        for (int shift = 0; shift < bits; shift += 8) {
            k_rs_count<<<(unsigned)nblocks, kRsThreads, 0, s>>>(key[cur], n, shift, hist);
            GBC_TRY(exclusive_scan_i64(ws, hist, hist, kRsRadix * nblocks, s));
            k_rs_scatter<<<(unsigned)nblocks, kRsThreads, 0, s>>>(key[cur], idx[cur], n, shift, hist, key[cur ^ 1],
                                                                   idx[cur ^ 1]);
            note_launches(2);
            cur ^= 1;
        }
    }
    // rows with entries, their starts
    if (p->tiles) {
        int64_t *index = nullptr;
        GBC_TRY(ws.alloc_n(&index, p->m + 1));
        const unsigned rg = (unsigned)((p->m + 255) / 256);
        if (p->m > 0) {
            k_spmv_has<<<rg, 256, 0, s>>>(p->m, p->rowptr, index);
            note_launch();
        }
        GBC_TRY(exclusive_scan_i64(ws, index, index, p->m, s));
        GBC_TRY(read_i64(ctx, index + p->m, &p->nrows));
        p->ntiles = (n + kSpmvTile - 1) / kSpmvTile;
        GBC_TRY(device_alloc(ctx, (void **)&p->rows, (p->nrows + 1) * sizeof(int32_t)));
        GBC_TRY(device_alloc(ctx, (void **)&p->starts, (n / 32 + 2) * sizeof(uint32_t)));
        GBC_TRY(device_alloc(ctx, (void **)&p->group_row, (n / kSpmvPer + 1) * sizeof(int32_t)));
        GBC_TRY(device_alloc(ctx, &p->edge, (2 * p->ntiles + 1) * sizeof(int64_t)));  // widest value type
        GBC_TRY(device_alloc(ctx, (void **)&p->edge_row, (p->ntiles + 1) * sizeof(int32_t)));
        GBC_CUDA_TRY(cudaMemsetAsync(p->starts, 0, (n / 32 + 2) * sizeof(uint32_t), s));
        if (p->m > 0) {
            k_spmv_mark<<<rg, 256, 0, s>>>(p->m, p->rowptr, index, p->rows, p->starts, p->group_row);
            note_launch();
        }
    }
    switch (p->vt) {
        case GBC_F64: GBC_TRY(plan_values<double>(p, ws, A, idx[cur], col_cm)); break;
        case GBC_F32: GBC_TRY(plan_values<float>(p, ws, A, idx[cur], col_cm)); break;
        case GBC_I64: GBC_TRY(plan_values<int64_t>(p, ws, A, idx[cur], col_cm)); break;
        case GBC_BOOL: GBC_TRY(plan_values<uint8_t>(p, ws, A, idx[cur], col_cm)); break;
        default: return fail(GBC_EINVAL, "unknown value type");
    }
    GBC_CUDA_TRY(cudaGetLastError());
    int32_t herr = 0;
    GBC_CUDA_TRY(cudaMemcpyAsync(&herr, err, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    GBC_CUDA_TRY(cudaStreamSynchronize(s));
    if (herr) return fail(GBC_EINVAL, "SpMV plan: row id out of range");
    return GBC_OK;
}

template <class SR>
static int spmv_run(SpmvPlan *p, const void *x, void *y)
{
    typedef typename SR::V V;
    cudaStream_t s = p->ctx->stream;
    if (p->ntiles == 0) return GBC_OK;
    k_spmv_tiles<SR><<<(unsigned)p->ntiles, kSpmvThreads, 0, s>>>(
        p->nnz, p->starts, p->group_row, p->rows, p->col, static_cast<const V *>(p->val), static_cast<const V *>(x),
        static_cast<V *>(y), static_cast<V *>(p->edge), p->edge_row);
    k_spmv_edges<SR><<<(unsigned)(p->ntiles / 128 + 1), 128, 0, s>>>(p->ntiles, p->nrows, p->rows,
                                                                     static_cast<const V *>(p->edge), p->edge_row,
                                                                     static_cast<V *>(y));
    note_launches(2);
    GBC_CUDA_TRY(cudaGetLastError());
    return GBC_OK;
}

void spmv_plan_release(SpmvPlan *p)
{
    if (!p->ctx) return;
    cudaSetDevice(p->ctx->device);
    cudaStreamSynchronize(p->ctx->stream);
    device_free(p->ctx, p->rowptr);
    device_free(p->ctx, p->col);
    device_free(p->ctx, p->val);
    device_free(p->ctx, p->rows);
    device_free(p->ctx, p->starts);
    device_free(p->ctx, p->group_row);
    device_free(p->ctx, p->edge);
    device_free(p->ctx, p->edge_row);
    cudaStreamSynchronize(p->ctx->stream);
}

}  // namespace gbc

using namespace gbc;

struct gbc_spmv_plan : gbc::SpmvPlan {};

extern "C" {

int gbc_spmv_plan_create(gbc_context *ctx, int vt, const gbc_matrix *A, gbc_spmv_plan **out)
{
    if (!ctx || !A || !out) return fail(GBC_EINVAL, "null argument");
    *out = nullptr;
    if (vt != GBC_F64 && vt != GBC_F32 && vt != GBC_I64 && vt != GBC_BOOL) return fail(GBC_EINVAL, "bad value type");
    GBC_CUDA_TRY(cudaSetDevice(ctx->device));
    gbc_spmv_plan *p = new gbc_spmv_plan();
    p->ctx = ctx;
    p->vt = vt;
    const int rc = spmv_plan_build(p, A);
    if (rc != GBC_OK) {
        gbc_spmv_plan_destroy(p);
        return rc;
    }
    *out = p;
    return GBC_OK;
}

int gbc_spmv_plan_destroy(gbc_spmv_plan *p)
{
    if (!p) return GBC_OK;
    spmv_plan_release(p);
    delete p;
    return GBC_OK;
}

int gbc_spmv(gbc_context *ctx, const gbc_spmv_plan *p, int sr, const void *x, void *y, int where)
{
    if (!ctx || !p || !x || !y) return fail(GBC_EINVAL, "null argument");
    if (where != GBC_HOST && where != GBC_DEVICE) return fail(GBC_EINVAL, "bad memory location");
    GBC_CUDA_TRY(cudaSetDevice(ctx->device));
    SpmvPlan *q = const_cast<gbc_spmv_plan *>(p);
    q->ctx = ctx;
    cudaStream_t s = ctx->stream;
    const size_t vs = value_size(p->vt);
    Workspace ws(ctx);
    const void *dx = x;
    void *dy = y;
    if (where == GBC_HOST) {
        void *bx = nullptr, *by = nullptr;
        GBC_TRY(ws.alloc(&bx, p->n * vs + 16));
        GBC_TRY(ws.alloc(&by, p->m * vs + 16));
        GBC_CUDA_TRY(cudaMemcpyAsync(bx, x, p->n * vs, cudaMemcpyHostToDevice, s));
        GBC_CUDA_TRY(cudaMemcpyAsync(by, y, p->m * vs, cudaMemcpyHostToDevice, s));
        dx = bx;
        dy = by;
    }
    int rc = fail(GBC_EUNSUPPORTED, "semiring/value type combination not instantiated");
    switch (sr) {
        case GBC_SR_PLUSTIMES:
            if (p->vt == GBC_F64) rc = spmv_run<PlusTimes<double>>(q, dx, dy);
            if (p->vt == GBC_F32) rc = spmv_run<PlusTimes<float>>(q, dx, dy);
            if (p->vt == GBC_I64) rc = spmv_run<PlusTimes<int64_t>>(q, dx, dy);
            if (p->vt == GBC_BOOL) rc = spmv_run<BoolOrAnd>(q, dx, dy);
            break;
        case GBC_SR_BOOL:
            if (p->vt == GBC_BOOL) rc = spmv_run<BoolOrAnd>(q, dx, dy);
            break;
        case GBC_SR_MINPLUS:
            if (p->vt == GBC_F64) rc = spmv_run<MinPlus<double>>(q, dx, dy);
            if (p->vt == GBC_I64) rc = spmv_run<MinPlus<int64_t>>(q, dx, dy);
            break;
        case GBC_SR_SELECT2NDMIN:
            if (p->vt == GBC_I64) rc = spmv_run<Select2ndMin<int64_t>>(q, dx, dy);
            break;
        default: break;
    }
    if (rc != GBC_OK) return rc;
    if (where == GBC_HOST) GBC_CUDA_TRY(cudaMemcpyAsync(y, dy, p->m * vs, cudaMemcpyDeviceToHost, s));
    GBC_CUDA_TRY(cudaStreamSynchronize(s));
    return GBC_OK;
}

}  // extern "C"
