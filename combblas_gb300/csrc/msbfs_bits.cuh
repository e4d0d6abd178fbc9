// Multi-source BFS with one bit per root (included by spmspv.cu).
//
// The Select2ndMin product over all roots at once takes, for a vertex v and
// every root that has not reached it, the smallest neighbour of v in that
// root's frontier.  For a symmetric pattern whose columns are ascending, v's
// neighbours are its own column, in the order that the minimum asks for.  So a
// frontier is held as NW 64-bit words per vertex (up to 64 NW roots), and one
// pass over the edges serves all roots: a lane owns 64 roots of one vertex,
// walks the neighbours, and the first one whose frontier word has a wanted
// bit is that root's parent.  Per edge and level that is one 4-byte id and one
// 8 NW-byte gather, instead of one visited test, one candidate test and one
// atomic per edge, root and level.  R-MAT scale 20, 256 roots: 122.6 ms by
// (root, vertex) pairs, 6.7 ms here, bound by the parents' scattered 8-byte
// stores and the frontier gathers from L2.
//
// A level runs in one of two ways, chosen on the device from the edges of the
// active vertices (those with a bit in the frontier):
//   pull  all vertices look for their parents as above.  Vertices of more than
//         kMbChunk neighbours are cut into chunks, whose parents meet in an
//         atomic minimum (an unreached parent, -1, is the largest unsigned).
//   push  the active vertices' edges only: neighbours' words by atomicOr,
//         parents by atomic minimum.  Everything a push level touches is in its
//         two vertex lists, so long thin graphs pay for their frontiers only.
#pragma once

#include "size_rules.cuh"

namespace gbc {

constexpr int kMbWords = 8;      // 512 roots a pass
constexpr int kMbChunk = 64;     // neighbours of one pull item
constexpr int kMbPullShare = 4;  // pull when the active edges times this exceed all edges
constexpr int kMbPushThreads = 128;  // a block of k_mb_push, and its step over a long vertex
static_assert(kMbPushThreads <= kMbStep && kMbChunk <= kMbStep, "mb_positions_fit");

enum {
    MB_NF = 0,       // active vertices
    MB_NNEXT = 1,    // active vertices of the next frontier
    MB_LEVEL = 2,    // levels of this pass
    MB_FE = 3,       // edges of the active vertices
    MB_FE_NEXT = 4,
    MB_MODE = 5,     // 0 push, 1 pull
    MB_CUR = 6,      // which frontier buffer and list is current
    MB_ROOTS = 7,    // roots of this pass
    MB_PARENTS = 8,  // parents of its first root (address)
    MB_EDGES = 9,    // over all passes: sum of degrees of reached pairs,
    MB_REACHED = 10, //   reached pairs,
    MB_LEVELS = 11,  //   the most levels of a pass
    MB_N = 16
};

struct MbView {
    const uint32_t *cp;
    const int32_t *row;
    int64_t n, nnz;
    int64_t *ctl;
    uint64_t *seen;
    uint64_t *bits0, *bits1;
    int32_t *list0, *list1;
    uint32_t *touched;
    __device__ __forceinline__ uint64_t *bits(int k) const { return k ? bits1 : bits0; }
    __device__ __forceinline__ int32_t *list(int k) const { return k ? list1 : list0; }
    const int32_t *item_v;   // pull chunks of the long vertices
    const uint32_t *item_p;  //   ... and where they start
    int64_t nitems;
};

// Entries below the diagonal must have their mirror image, and there must be
// as many above: then the pattern is symmetric.  Columns must be strictly
// ascending.  out: [0] a fault, [1] entries above, [2] below the diagonal.
__global__ void k_mb_check(int64_t n, const uint32_t *cp, const int32_t *row, unsigned long long *out)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
    unsigned long long above = 0, below = 0;
    bool bad = false;
    for (int64_t c = warp; c < n; c += nwarps) {
        const uint32_t s = cp[c], e = cp[c + 1];
        for (uint32_t p = s + lane; p < e; p += 32) {
            const int32_t r = row[p];
            if (p > s && row[p - 1] >= r) bad = true;
            if (r < c) ++above;
            if (r > c) {
                ++below;
                uint32_t lo = cp[r], hi = cp[r + 1];
                const uint32_t end = hi;
                while (lo < hi) {
                    const uint32_t mid = lo + (hi - lo) / 2;
                    if (row[mid] < (int32_t)c)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                if (lo >= end || row[lo] != (int32_t)c) bad = true;
            }
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        above += __shfl_xor_sync(0xffffffffu, above, o);
        below += __shfl_xor_sync(0xffffffffu, below, o);
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
        if (bad) atomicOr(&out[0], 1ull);
        if (above) atomicAdd(&out[1], above);
        if (below) atomicAdd(&out[2], below);
    }
}

// Pull chunks of the vertices of more than kMbChunk neighbours: counted
// (item_v null), or filled in.
__global__ void k_mb_items(int64_t n, const uint32_t *cp, unsigned long long *count, int32_t *item_v,
                           uint32_t *item_p)
{
    const int64_t v = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const uint32_t s = cp[v], d = cp[v + 1] - s;
    if (d <= kMbChunk) return;
    const uint32_t k = (d + kMbChunk - 1) / kMbChunk;
    const unsigned long long o = atomicAdd(count, (unsigned long long)k);
    if (item_v)
        for (uint32_t i = 0; i < k; ++i) {
            item_v[o + i] = (int32_t)v;
            item_p[o + i] = s + i * kMbChunk;
        }
}

template <int NW>
__global__ void k_mb_init(MbView g, const int64_t *roots, int64_t nroots, int64_t *parents)
{
    const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (r == 0) {
        g.ctl[MB_ROOTS] = nroots;
        g.ctl[MB_PARENTS] = (int64_t)(uintptr_t)parents;
    }
    if (r >= nroots) return;
    const int64_t v = roots[r];
    const unsigned long long bit = 1ull << (r & 63);
    parents[r * g.n + v] = v;
    atomicOr((unsigned long long *)&g.seen[v * NW + (r >> 6)], bit);
    atomicOr((unsigned long long *)&g.bits(0)[v * NW + (r >> 6)], bit);
    const unsigned long long d = g.cp[v + 1] - g.cp[v];
    if (!(atomicOr(&g.touched[v >> 5], 1u << (v & 31)) & (1u << (v & 31)))) {
        g.list(0)[atomicAdd((unsigned long long *)&g.ctl[MB_NF], 1ull)] = (int32_t)v;
        atomicAdd((unsigned long long *)&g.ctl[MB_FE], d);
    }
    atomicAdd((unsigned long long *)&g.ctl[MB_EDGES], d);
    atomicAdd((unsigned long long *)&g.ctl[MB_REACHED], 1ull);
}

__device__ __forceinline__ void mb_mode(int64_t *ctl, int64_t nnz)
{
    ctl[MB_MODE] = ctl[MB_FE] * kMbPullShare > nnz ? 1 : 0;
}

// The roots' touched marks are cleared, the first level's mode is chosen.
__global__ void k_mb_begin(MbView g)
{
    for (int64_t i = threadIdx.x; i < g.ctl[MB_NF]; i += blockDim.x) g.touched[g.list(0)[i] >> 5] = 0;
    if (threadIdx.x == 0) mb_mode(g.ctl, g.nnz);
}

// Push: a warp per active vertex, the block together for the long ones.
template <int NW>
__global__ void __launch_bounds__(kMbPushThreads) k_mb_push(MbView g)
{
    if (g.ctl[MB_MODE] != 0) return;
    __shared__ int32_t s_long[4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t nf = g.ctl[MB_NF];
    const int cur = (int)g.ctl[MB_CUR];
    const uint64_t *front = g.bits(cur);
    uint64_t *next = g.bits(cur ^ 1);
    int32_t *nlist = g.list(cur ^ 1);
    unsigned long long *parents = (unsigned long long *)(uintptr_t)g.ctl[MB_PARENTS];
    auto edges = [&](int32_t u, int first, int step) {
        uint64_t f[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) f[w] = front[(int64_t)u * NW + w];
        const uint32_t s = g.cp[u], e = g.cp[u + 1];
        for (uint32_t p = s + first; p < e; p += step) {
            const int32_t v = g.row[p];
            bool any = false;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                if (f[w] == 0) continue;
                uint64_t x = f[w] & ~g.seen[(int64_t)v * NW + w];
                if (x == 0) continue;
                any = true;
                atomicOr((unsigned long long *)&next[(int64_t)v * NW + w], (unsigned long long)x);
                while (x) {
                    const int b = __ffsll((long long)x) - 1;
                    x &= x - 1;
                    atomicMin(&parents[(int64_t)(w * 64 + b) * g.n + v], (unsigned long long)u);
                }
            }
            if (any && !(atomicOr(&g.touched[v >> 5], 1u << (v & 31)) & (1u << (v & 31))))
                nlist[atomicAdd((unsigned long long *)&g.ctl[MB_NNEXT], 1ull)] = v;
        }
    };
    for (int64_t b = int64_t(blockIdx.x) * 4; b < nf; b += int64_t(gridDim.x) * 4) {
        int32_t u = -1;
        if (b + warp < nf) u = g.list(cur)[b + warp];
        const bool is_long = u >= 0 && g.cp[u + 1] - g.cp[u] > 512;
        if (lane == 0) s_long[warp] = is_long ? u : -1;
        if (u >= 0 && !is_long) edges(u, lane, 32);
        __syncthreads();
        for (int k = 0; k < 4; ++k)
            if (s_long[k] >= 0) edges(s_long[k], threadIdx.x, kMbPushThreads);
        __syncthreads();
    }
}

__device__ __forceinline__ void mb_count(int64_t *ctl, unsigned long long reached, unsigned long long deg,
                                         unsigned long long fe)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        reached += __shfl_xor_sync(0xffffffffu, reached, o);
        deg += __shfl_xor_sync(0xffffffffu, deg, o);
        fe += __shfl_xor_sync(0xffffffffu, fe, o);
    }
    if ((threadIdx.x & 31) == 0 && (reached || fe)) {
        atomicAdd((unsigned long long *)&ctl[MB_REACHED], reached);
        atomicAdd((unsigned long long *)&ctl[MB_EDGES], deg);
        atomicAdd((unsigned long long *)&ctl[MB_FE_NEXT], fe);
    }
}

// End of a push level: the new vertices' bits are seen, the old frontier's
// buffer is zero again.
template <int NW>
__global__ void __launch_bounds__(256) k_mb_push_end(MbView g)
{
    if (g.ctl[MB_MODE] != 0) return;
    const int cur = (int)g.ctl[MB_CUR];
    const int64_t i0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, stride = int64_t(gridDim.x) * blockDim.x;
    const int64_t nn = g.ctl[MB_NNEXT], nf = g.ctl[MB_NF];
    unsigned long long reached = 0, deg = 0, fe = 0;
    for (int64_t i = i0; i < nn; i += stride) {
        const int64_t v = g.list(cur ^ 1)[i];
        g.touched[v >> 5] = 0;
        const unsigned long long d = g.cp[v + 1] - g.cp[v];
        int c = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const uint64_t x = g.bits(cur ^ 1)[v * NW + w];
            if (x) g.seen[v * NW + w] |= x;
            c += __popcll(x);
        }
        reached += c;
        deg += c * d;
        fe += d;
    }
    for (int64_t i = i0; i < nf; i += stride) {
        const int64_t v = g.list(cur)[i];
#pragma unroll
        for (int w = 0; w < NW; ++w) g.bits(cur)[v * NW + w] = 0;
    }
    mb_count(g.ctl, reached, deg, fe);
}

// Pull: NW lanes per item (a short vertex, or a chunk of a long one).
template <int NW>
__global__ void __launch_bounds__(256) k_mb_pull(MbView g)
{
    if (g.ctl[MB_MODE] != 1) return;
    constexpr int U = 4;  // neighbours in flight
    const int w = threadIdx.x % NW;
    const int cur = (int)g.ctl[MB_CUR];
    const uint64_t *front = g.bits(cur);
    uint64_t *next = g.bits(cur ^ 1);
    unsigned long long *parents = (unsigned long long *)(uintptr_t)g.ctl[MB_PARENTS] + (int64_t)w * 64 * g.n;
    const int64_t left = g.ctl[MB_ROOTS] - w * 64;
    const uint64_t valid = left >= 64 ? ~0ull : left > 0 ? (1ull << left) - 1 : 0ull;
    const int64_t stride = int64_t(gridDim.x) * (256 / NW);
    for (int64_t i = int64_t(blockIdx.x) * (256 / NW) + threadIdx.x / NW; i < g.nitems + g.n; i += stride) {
        const bool chunk = i < g.nitems;
        const int64_t v = chunk ? g.item_v[i] : i - g.nitems;
        uint32_t p = chunk ? g.item_p[i] : g.cp[v], e = g.cp[v + 1];
        if (chunk)
            e = min(e, p + kMbChunk);
        else if (e - p > kMbChunk)
            continue;  // its chunks are items of their own
        uint64_t want = valid & ~g.seen[v * NW + w], found = 0;
        for (; p < e && want; p += U) {
            int32_t u[U];
            uint64_t f[U];
#pragma unroll
            for (int k = 0; k < U; ++k) u[k] = p + k < e ? g.row[p + k] : -1;
#pragma unroll
            for (int k = 0; k < U; ++k) f[k] = u[k] >= 0 ? front[(int64_t)u[k] * NW + w] : 0ull;
#pragma unroll
            for (int k = 0; k < U; ++k) {
                uint64_t x = f[k] & want;
                want &= ~x;
                found |= x;
                while (x) {
                    unsigned long long *at = &parents[(int64_t)(__ffsll((long long)x) - 1) * g.n + v];
                    x &= x - 1;
                    if (chunk)
                        atomicMin(at, (unsigned long long)u[k]);
                    else
                        *at = (unsigned long long)u[k];
                }
            }
        }
        if (found) {
            if (chunk)
                atomicOr((unsigned long long *)&next[v * NW + w], (unsigned long long)found);
            else
                next[v * NW + w] = found;
        }
    }
}

// End of a pull level, over all vertices: as k_mb_push_end, and the next
// frontier's list.
template <int NW>
__global__ void __launch_bounds__(256) k_mb_pull_end(MbView g)
{
    if (g.ctl[MB_MODE] != 1) return;
    const int cur = (int)g.ctl[MB_CUR], lane = threadIdx.x & 31;
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    unsigned long long reached = 0, deg = 0, fe = 0;
    for (int64_t b = int64_t(blockIdx.x) * blockDim.x; b < g.n; b += stride) {
        const int64_t v = b + threadIdx.x;
        int c = 0;
        if (v < g.n) {
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const uint64_t x = g.bits(cur ^ 1)[v * NW + w];
                if (x) g.seen[v * NW + w] |= x;
                c += __popcll(x);
                g.bits(cur)[v * NW + w] = 0;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, c > 0);
        if (m) {
            unsigned long long o = 0;
            if (lane == 0) o = atomicAdd((unsigned long long *)&g.ctl[MB_NNEXT], (unsigned long long)__popc(m));
            o = __shfl_sync(0xffffffffu, o, 0);
            if (c > 0) {
                const unsigned long long d = g.cp[v + 1] - g.cp[v];
                g.list(cur ^ 1)[o + __popc(m & ((1u << lane) - 1))] = (int32_t)v;
                reached += c;
                deg += c * d;
                fe += d;
            }
        }
    }
    mb_count(g.ctl, reached, deg, fe);
}

__global__ void k_mb_advance(int64_t *ctl, int64_t nnz, int64_t cap, cudaGraphConditionalHandle h)
{
    ctl[MB_NF] = ctl[MB_NNEXT];
    ctl[MB_NNEXT] = 0;
    ctl[MB_FE] = ctl[MB_FE_NEXT];
    ctl[MB_FE_NEXT] = 0;
    ctl[MB_CUR] ^= 1;
    ctl[MB_LEVEL] += 1;
    if (ctl[MB_LEVEL] > ctl[MB_LEVELS]) ctl[MB_LEVELS] = ctl[MB_LEVEL];
    mb_mode(ctl, nnz);
    cudaGraphSetConditional(h, (ctl[MB_NF] != 0 && ctl[MB_LEVEL] < cap) ? 1u : 0u);
}

static MbView mb_view(const Graph *g)
{
    const MsBits &b = g->mb;
    MbView v;
    v.cp = g->cp32;
    v.row = g->row;
    v.n = g->n;
    v.nnz = g->nnz;
    v.ctl = b.ctl;
    v.seen = b.seen;
    v.bits0 = b.bits[0];
    v.bits1 = b.bits[1];
    v.list0 = b.list[0];
    v.list1 = b.list[1];
    v.touched = b.touched;
    v.item_v = b.item_v;
    v.item_p = b.item_p;
    v.nitems = b.nitems;
    return v;
}

static void mb_free(Graph *g)
{
    MsBits &b = g->mb;
    Context *c = g->ctx;
    for (auto &e : b.exec) {
        if (e) cudaGraphExecDestroy(e);
        e = nullptr;
    }
    device_free(c, b.seen);
    device_free(c, b.bits[0]);
    device_free(c, b.bits[1]);
    device_free(c, b.list[0]);
    device_free(c, b.list[1]);
    device_free(c, b.touched);
    device_free(c, b.ctl);
    device_free(c, b.item_v);
    device_free(c, b.item_p);
    if (b.h_ctl) cudaFreeHost(b.h_ctl);
    const int form = b.form;
    b = MsBits();
    b.form = form;
}

// Whether the graph is symmetric with ascending columns (looked at once; the
// graph's arrays are its own and never change), and the pull chunks.
static int mb_prepare(Graph *g)
{
    MsBits &b = g->mb;
    Context *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    if (b.form == 0 && !mb_positions_fit(g->nnz)) b.form = 2;
    if (b.form == 2 || b.list[0]) return GBC_OK;
    if (b.form == 0) {
        Workspace ws(ctx);
        unsigned long long *out = nullptr, h[3] = {0, 0, 0};
        GBC_TRY(ws.alloc_n(&out, 4));
        GBC_CUDA_TRY(cudaMemsetAsync(out, 0, 4 * sizeof(unsigned long long), s));
        if (g->n > 0) {
            k_mb_check<<<ctx->num_sms * 8, 256, 0, s>>>(g->n, g->cp32, g->row, out);
            note_launch();
        }
        GBC_CUDA_TRY(cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, s));
        GBC_CUDA_TRY(cudaStreamSynchronize(s));
        b.form = (h[0] == 0 && h[1] == h[2]) ? 1 : 2;
        if (b.form == 2) return GBC_OK;
    }
    Workspace ws(ctx);
    unsigned long long *cnt = nullptr;
    GBC_TRY(ws.alloc_n(&cnt, 2));
    GBC_CUDA_TRY(cudaMemsetAsync(cnt, 0, 2 * sizeof(unsigned long long), s));
    const unsigned grid = (unsigned)((g->n + 255) / 256);
    k_mb_items<<<grid, 256, 0, s>>>(g->n, g->cp32, cnt, nullptr, nullptr);
    note_launch();
    GBC_TRY(read_i64(ctx, reinterpret_cast<const int64_t *>(cnt), &b.nitems));
    GBC_TRY(device_alloc(ctx, (void **)&b.item_v, (b.nitems + 1) * sizeof(int32_t)));
    GBC_TRY(device_alloc(ctx, (void **)&b.item_p, (b.nitems + 1) * sizeof(uint32_t)));
    if (b.nitems > 0) {
        k_mb_items<<<grid, 256, 0, s>>>(g->n, g->cp32, cnt + 1, b.item_v, b.item_p);
        note_launch();
    }
    GBC_TRY(device_alloc(ctx, (void **)&b.touched, (g->n / 32 + 1) * sizeof(uint32_t)));
    GBC_CUDA_TRY(cudaMemsetAsync(b.touched, 0, (g->n / 32 + 1) * sizeof(uint32_t), s));
    GBC_TRY(device_alloc(ctx, (void **)&b.ctl, MB_N * sizeof(int64_t)));
    GBC_CUDA_TRY(cudaMallocHost(&b.h_ctl, MB_N * sizeof(int64_t)));
    GBC_TRY(device_alloc(ctx, (void **)&b.list[1], (g->n + 1) * sizeof(int32_t)));
    GBC_TRY(device_alloc(ctx, (void **)&b.list[0], (g->n + 1) * sizeof(int32_t)));  // last: marks it ready
    return GBC_OK;
}

static int mb_reserve(Graph *g, int words)
{
    MsBits &b = g->mb;
    if (b.words >= words) return GBC_OK;
    Context *ctx = g->ctx;
    for (auto &e : b.exec) {  // their arrays move
        if (e) cudaGraphExecDestroy(e);
        e = nullptr;
    }
    device_free(ctx, b.seen);
    device_free(ctx, b.bits[0]);
    device_free(ctx, b.bits[1]);
    b.seen = b.bits[0] = b.bits[1] = nullptr;
    b.words = 0;
    const size_t bytes = (size_t)g->n * words * sizeof(uint64_t) + 16;
    GBC_TRY(device_alloc(ctx, (void **)&b.seen, bytes));
    GBC_TRY(device_alloc(ctx, (void **)&b.bits[0], bytes));
    GBC_TRY(device_alloc(ctx, (void **)&b.bits[1], bytes));
    b.words = words;
    return GBC_OK;
}

// One pass over at most 64 NW roots; nothing is read back.
template <int NW>
static int mb_pass(Graph *g, int slot, const int64_t *d_roots, int64_t nroots, int64_t *parents)
{
    MsBits &b = g->mb;
    Context *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    const MbView v = mb_view(g);
    if (!b.exec[slot]) {
        auto body = [&](cudaStream_t cs, cudaGraphConditionalHandle h) {
            k_mb_push<NW><<<occ_grid(ctx, (const void *)k_mb_push<NW>, kMbPushThreads, 0), kMbPushThreads, 0, cs>>>(v);
            k_mb_push_end<NW><<<occ_grid(ctx, (const void *)k_mb_push_end<NW>, 256, 0), 256, 0, cs>>>(v);
            k_mb_pull<NW><<<occ_grid(ctx, (const void *)k_mb_pull<NW>, 256, 0), 256, 0, cs>>>(v);
            k_mb_pull_end<NW><<<occ_grid(ctx, (const void *)k_mb_pull_end<NW>, 256, 0), 256, 0, cs>>>(v);
            k_mb_advance<<<1, 1, 0, cs>>>(v.ctl, v.nnz, v.n + 2, h);
            note_launches(5);
            GBC_CUDA_TRY(cudaGetLastError());
            return (int)GBC_OK;
        };
        // (a CUDA driver without conditional nodes)
        if (loop_graph(body, true, nullptr, nullptr, 0, &b.exec[slot], &b.kernels) != GBC_OK) return GBC_EUNSUPPORTED;
    }
    const size_t bytes = (size_t)g->n * NW * sizeof(uint64_t);
    GBC_CUDA_TRY(cudaMemsetAsync(b.seen, 0, bytes, s));
    GBC_CUDA_TRY(cudaMemsetAsync(b.bits[0], 0, bytes, s));
    GBC_CUDA_TRY(cudaMemsetAsync(b.bits[1], 0, bytes, s));
    GBC_CUDA_TRY(cudaMemsetAsync(b.ctl, 0, MB_EDGES * sizeof(int64_t), s));
    k_mb_init<NW><<<(unsigned)((nroots + 255) / 256), 256, 0, s>>>(v, d_roots, nroots, parents);
    k_mb_begin<<<1, 256, 0, s>>>(v);
    note_launches(2);
    GBC_CUDA_TRY(cudaGetLastError());
    GBC_CUDA_TRY(cudaGraphLaunch(b.exec[slot], s));
    return GBC_OK;
}

// parents: device [nroots * n], root-major.  The graph is prepared (form 1).
// GBC_EUNSUPPORTED: the traversal graph cannot be built.
static int mb_msbfs(Graph *g, const int64_t *d_roots, int64_t nroots, int64_t *parents, gbc_msbfs_stats *st)
{
    MsBits &b = g->mb;
    Context *ctx = g->ctx;
    cudaStream_t s = ctx->stream;
    const int64_t most = std::min<int64_t>(nroots, 64 * kMbWords);
    GBC_TRY(mb_reserve(g, most <= 64 ? 1 : most <= 128 ? 2 : most <= 256 ? 4 : 8));
    cudaEventRecord(ctx->ev[5], s);
    GBC_CUDA_TRY(cudaMemsetAsync(parents, 0xff, nroots * g->n * sizeof(int64_t), s));  // -1: unreached
    GBC_CUDA_TRY(cudaMemsetAsync(b.ctl, 0, MB_N * sizeof(int64_t), s));
    for (int64_t r0 = 0; r0 < nroots; r0 += 64 * kMbWords) {
        const int64_t nr = std::min<int64_t>(nroots - r0, 64 * kMbWords);
        int64_t *dp = parents + r0 * g->n;
        if (nr <= 64)
            GBC_TRY(mb_pass<1>(g, 0, d_roots + r0, nr, dp));
        else if (nr <= 128)
            GBC_TRY(mb_pass<2>(g, 1, d_roots + r0, nr, dp));
        else if (nr <= 256)
            GBC_TRY(mb_pass<4>(g, 2, d_roots + r0, nr, dp));
        else
            GBC_TRY(mb_pass<8>(g, 3, d_roots + r0, nr, dp));
    }
    GBC_CUDA_TRY(cudaMemcpyAsync(b.h_ctl, b.ctl, MB_N * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    cudaEventRecord(ctx->ev[6], s);
    GBC_CUDA_TRY(cudaEventSynchronize(ctx->ev[6]));
    note_launches(b.kernels * std::max<int64_t>(b.h_ctl[MB_LEVELS], 1));
    if (st) {
        float ms = 0;
        cudaEventElapsedTime(&ms, ctx->ev[5], ctx->ev[6]);
        st->levels = b.h_ctl[MB_LEVELS];
        st->reached = b.h_ctl[MB_REACHED];
        st->edges = b.h_ctl[MB_EDGES] / 2;
        st->ms = ms;
        st->host_checks = 0;
    }
    return GBC_OK;
}

}  // namespace gbc
