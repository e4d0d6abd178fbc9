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
//         A block flattens the edges of a few vertices over its threads; the
//         hubs, of more than kMbHub neighbours, are listed apart and shared out over
//         groups of blocks.
#pragma once

#include "size_rules.cuh"

namespace gbc {

constexpr int kMbWords = 8;      // 512 roots a pass
constexpr int kMbChunk = 64;     // neighbours of one pull item
constexpr int kMbPullShare = 4;  // pull when the active edges times this exceed all edges
static_assert(kMbChunk <= kMbStep, "mb_positions_fit");
constexpr int kMbQueue = 1024;   // new vertices that a block gathers before it lists them
constexpr int kMbThreads = 256;  // of a block, and the vertices it pushes at most at a time
constexpr uint32_t kMbHub = 2048;

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
    MB_NHUB = 9,     // hubs among the active vertices
    MB_NHUB_NEXT = 10,
    MB_EDGES = 11,   // over all passes: sum of degrees of reached pairs,
    MB_REACHED = 12, //   reached pairs,
    MB_LEVELS = 13,  //   the most levels of a pass
    MB_DONE = 14,    // blocks that have ended the level
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
    int32_t *hubs0, *hubs1;
    uint32_t *touched;
    __device__ __forceinline__ uint64_t *bits(int k) const { return k ? bits1 : bits0; }
    __device__ __forceinline__ int32_t *list(int k) const { return k ? list1 : list0; }
    __device__ __forceinline__ int32_t *hubs(int k) const { return k ? hubs1 : hubs0; }
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
        if (d > kMbHub) g.hubs(0)[atomicAdd((unsigned long long *)&g.ctl[MB_NHUB], 1ull)] = (int32_t)v;
        atomicAdd((unsigned long long *)&g.ctl[MB_FE], d);
    }
    atomicAdd((unsigned long long *)&g.ctl[MB_EDGES], d);
    atomicAdd((unsigned long long *)&g.ctl[MB_REACHED], 1ull);
}

__device__ __forceinline__ int64_t mb_mode(int64_t fe, int64_t nnz) { return fe * kMbPullShare > nnz ? 1 : 0; }

// The roots' touched marks are cleared, the first level's mode is chosen.
__global__ void k_mb_begin(MbView g)
{
    for (int64_t i = threadIdx.x; i < g.ctl[MB_NF]; i += blockDim.x) g.touched[g.list(0)[i] >> 5] = 0;
    if (threadIdx.x == 0) g.ctl[MB_MODE] = mb_mode(g.ctl[MB_FE], g.nnz);
}

// New vertices of a block on their way to the next frontier's list, one atomic on
// its length per batch (one per warp: 700 x 700 grid with 500 roots 101 -> 81 ms, one
// root on 2^22 random vertices 1.35 -> 0.88).  Every thread of the block calls add()
// and step(); step() ends a round of at most NT vertices, end() the kernel.
template <int NT>
struct MbQueue {
    int32_t v[kMbQueue];
    int n;
    unsigned long long base;
    __device__ __forceinline__ void begin()
    {
        if (threadIdx.x == 0) n = 0;
        __syncthreads();
    }
    __device__ __forceinline__ void add(bool act, int32_t x)
    {
        const int lane = threadIdx.x & 31;
        const unsigned m = __ballot_sync(0xffffffffu, act);
        if (m == 0) return;
        int at = 0;
        if (lane == __ffs(m) - 1) at = atomicAdd(&n, __popc(m));
        at = __shfl_sync(0xffffffffu, at, __ffs(m) - 1);
        if (act) v[at + __popc(m & ((1u << lane) - 1))] = x;
    }
    __device__ __forceinline__ void flush(int64_t *ctl, int32_t *list)  // behind a barrier
    {
        const int have = n;
        if (threadIdx.x == 0 && have > 0)
            base = atomicAdd((unsigned long long *)&ctl[MB_NNEXT], (unsigned long long)have);
        __syncthreads();
        for (int k = threadIdx.x; k < have; k += NT) list[base + k] = v[k];
        __syncthreads();
    }
    __device__ __forceinline__ void step(int64_t *ctl, int32_t *list)
    {
        // (one thread looks, before the others of the round may have added: all decide alike)
        if (!__syncthreads_or(threadIdx.x == 0 && n > kMbQueue - 2 * NT)) return;
        flush(ctl, list);
        begin();
    }
    __device__ __forceinline__ void end(int64_t *ctl, int32_t *list)
    {
        __syncthreads();
        flush(ctl, list);
    }
};

// Push.  The vertices that a block takes at a time are as many as share the
// frontier out evenly, so that thin frontiers keep all blocks busy and wide ones
// of few neighbours all lanes.  Bound by the latency of an edge's chain (neighbour,
// its seen word, the atomics).  With a warp per vertex (a block above 512
// neighbours), an atomic per listed vertex and five launches a level: 700 x 700 grid
// with 500 roots 112 -> 81 ms, hubs of 300 on a path with 300 roots 228 -> 92, one
// root on 2^22 vertices with a hub of 10^6 neighbours 16.9 -> 0.58, without the hub
// 2.08 -> 0.84.
template <int NW>
__device__ __forceinline__ void mb_push(const MbView &g)
{
    constexpr int NT = kMbThreads;
    __shared__ int32_t s_u[NT];
    __shared__ uint32_t s_st[NT];
    __shared__ int32_t s_off[NT + 1];
    __shared__ MbQueue<NT> queue;
    const int tid = threadIdx.x;
    const int64_t nf = g.ctl[MB_NF], nh = g.ctl[MB_NHUB];
    const int cur = (int)g.ctl[MB_CUR];
    const uint64_t *front = g.bits(cur);
    uint64_t *next = g.bits(cur ^ 1);
    int32_t *nlist = g.list(cur ^ 1);
    unsigned long long *parents = (unsigned long long *)(uintptr_t)g.ctl[MB_PARENTS];
    // the edge from u to the entry at p (act: there is one); all threads
    auto edge = [&](bool act, int32_t u, uint32_t p) {
        bool fresh = false;
        int32_t v = 0;
        if (act) {
            v = g.row[p];
            uint64_t x[NW];
            bool any = false;
#pragma unroll
            for (int w = 0; w < NW; ++w) x[w] = front[(int64_t)u * NW + w];
#pragma unroll
            for (int w = 0; w < NW; ++w)
                if (x[w]) x[w] &= ~g.seen[(int64_t)v * NW + w];  // (few words, where there are many)
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                if (x[w] == 0) continue;
                any = true;
                atomicOr((unsigned long long *)&next[(int64_t)v * NW + w], (unsigned long long)x[w]);
                for (uint64_t y = x[w]; y; y &= y - 1)
                    atomicMin(&parents[(int64_t)(w * 64 + __ffsll((long long)y) - 1) * g.n + v],
                              (unsigned long long)u);
            }
            const uint32_t bit = 1u << (v & 31);
            fresh = any && !(g.touched[v >> 5] & bit) && !(atomicOr(&g.touched[v >> 5], bit) & bit);
        }
        queue.add(fresh, v);
        if (fresh && g.cp[v + 1] - g.cp[v] > kMbHub)
            g.hubs(cur ^ 1)[atomicAdd((unsigned long long *)&g.ctl[MB_NHUB_NEXT], 1ull)] = v;
        queue.step(g.ctl, nlist);
    };
    queue.begin();
    // hubs: groups of at least eight blocks take them in turn, a block its share of each
    if (nh > 0) {
        const int groups = (int)min(nh, (int64_t)max(gridDim.x / 8, 1u)), blocks = (int)gridDim.x / groups;
        const int group = (int)blockIdx.x / blocks, share = (int)blockIdx.x % blocks;
        for (int64_t h = group; group < groups && h < nh; h += groups) {
            const int32_t u = g.hubs(cur)[h];
            const uint32_t s = g.cp[u], d = g.cp[u + 1] - s;
            for (int64_t e0 = int64_t(share) * NT; e0 < d; e0 += int64_t(blocks) * NT)
                edge(e0 + tid < d, u, s + (uint32_t)(e0 + tid));
        }
    }
    const int per = (int)min(max(nf / gridDim.x, (int64_t)1), (int64_t)NT);
    if (per == 1) {
        for (int64_t b = blockIdx.x; b < nf; b += gridDim.x) {
            const int32_t u = g.list(cur)[b];
            const uint32_t s = g.cp[u], d = g.cp[u + 1] - s;
            for (uint32_t e0 = 0; e0 < d && d <= kMbHub; e0 += NT) edge(e0 + tid < d, u, s + e0 + tid);
        }
        queue.end(g.ctl, nlist);
        return;
    }
    for (int64_t b = int64_t(blockIdx.x) * per; b < nf; b += int64_t(gridDim.x) * per) {
        const int n = (int)min((int64_t)per, nf - b);
        int d = 0;
        if (tid < n) {
            const int32_t u = g.list(cur)[b + tid];
            const uint32_t s = g.cp[u], du = g.cp[u + 1] - s;
            s_u[tid] = u;
            s_st[tid] = s;
            d = du > kMbHub ? 0 : (int)du;
        }
        int64_t tot;
        const int off = (int)block_exclusive_sum64<NT>(d, &tot);
        s_off[tid] = off;
        if (tid == NT - 1) s_off[NT] = (int)tot;
        __syncthreads();
        for (int e0 = 0; e0 < (int)tot; e0 += NT) {
            const int e = e0 + tid;
            int lo = 0;
#pragma unroll
            for (int step = NT / 2; step; step >>= 1)
                if (s_off[lo + step] <= e) lo += step;
            edge(e < (int)tot, s_u[lo], s_st[lo] + (uint32_t)(e - s_off[lo]));
        }
        __syncthreads();
    }
    queue.end(g.ctl, nlist);
}

// A block's share of the level's sums (all its threads call it).
__device__ void mb_count(int64_t *ctl, unsigned long long reached, unsigned long long deg, unsigned long long fe)
{
    __shared__ unsigned long long s_sum[3];
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        reached += __shfl_xor_sync(0xffffffffu, reached, o);
        deg += __shfl_xor_sync(0xffffffffu, deg, o);
        fe += __shfl_xor_sync(0xffffffffu, fe, o);
    }
    if ((threadIdx.x & 31) == 0 && (reached || fe)) {
        atomicAdd(&s_sum[0], reached);
        atomicAdd(&s_sum[1], deg);
        atomicAdd(&s_sum[2], fe);
    }
    __syncthreads();
    if (threadIdx.x < 3 && s_sum[threadIdx.x])
        atomicAdd((unsigned long long *)&ctl[threadIdx.x == 0   ? MB_REACHED
                                             : threadIdx.x == 1 ? MB_EDGES
                                                                : MB_FE_NEXT],
                  s_sum[threadIdx.x]);
}

// End of a push level: the new vertices' bits are seen, the old frontier's
// buffer is zero again.
template <int NW>
__device__ __forceinline__ void mb_push_end(const MbView &g)
{
    const int cur = (int)g.ctl[MB_CUR];
    const int64_t i0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, stride = int64_t(gridDim.x) * blockDim.x;
    const int64_t nn = g.ctl[MB_NNEXT], nf = g.ctl[MB_NF];
    unsigned long long reached = 0, deg = 0, fe = 0;
    // a lane per word
    for (int64_t i = i0; i < nn * NW; i += stride) {
        const int64_t v = g.list(cur ^ 1)[i / NW], at = v * NW + i % NW;
        const unsigned long long d = g.cp[v + 1] - g.cp[v];
        const uint64_t x = g.bits(cur ^ 1)[at];
        if (x) g.seen[at] |= x;
        const int c = __popcll(x);
        reached += c;
        deg += c * d;
        if (i % NW == 0) {
            g.touched[v >> 5] = 0;
            fe += d;
        }
    }
    for (int64_t i = i0; i < nf * NW; i += stride) g.bits(cur)[g.list(cur)[i / NW] * (int64_t)NW + i % NW] = 0;
    mb_count(g.ctl, reached, deg, fe);
}

// Pull: NW lanes per item (a short vertex, or a chunk of a long one).
template <int NW>
__device__ __forceinline__ void mb_pull(const MbView &g)
{
    constexpr int U = 4;  // neighbours in flight
    const int w = threadIdx.x % NW;
    const int cur = (int)g.ctl[MB_CUR];
    const uint64_t *front = g.bits(cur);
    uint64_t *next = g.bits(cur ^ 1);
    unsigned long long *parents = (unsigned long long *)(uintptr_t)g.ctl[MB_PARENTS] + (int64_t)w * 64 * g.n;
    const int64_t left = g.ctl[MB_ROOTS] - w * 64;
    const uint64_t valid = left >= 64 ? ~0ull : left > 0 ? (1ull << left) - 1 : 0ull;
    const int64_t stride = int64_t(gridDim.x) * (kMbThreads / NW);
    for (int64_t i = int64_t(blockIdx.x) * (kMbThreads / NW) + threadIdx.x / NW; i < g.nitems + g.n; i += stride) {
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

// End of a pull level, over all vertices: as mb_push_end, and the next
// frontier's list.
template <int NW>
__device__ __forceinline__ void mb_pull_end(const MbView &g)
{
    __shared__ MbQueue<kMbThreads> queue;
    const int cur = (int)g.ctl[MB_CUR];
    const int64_t stride = int64_t(gridDim.x) * blockDim.x;
    unsigned long long reached = 0, deg = 0, fe = 0;
    queue.begin();
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
        if (c > 0) {
            const unsigned long long d = g.cp[v + 1] - g.cp[v];
            if (d > kMbHub) g.hubs(cur ^ 1)[atomicAdd((unsigned long long *)&g.ctl[MB_NHUB_NEXT], 1ull)] = (int32_t)v;
            reached += c;
            deg += c * d;
            fe += d;
        }
        queue.add(c > 0, (int32_t)v);
        queue.step(g.ctl, g.list(cur ^ 1));
    }
    queue.end(g.ctl, g.list(cur ^ 1));
    mb_count(g.ctl, reached, deg, fe);
}

// A level is two launches, each of them one way or the other: with an idle
// kernel for the other way, and one to advance, a level of a thin frontier was
// mostly launches (20000 levels of a path 267 -> 217 ms).
template <int NW>
__global__ void __launch_bounds__(kMbThreads) k_mb_level(MbView g)
{
    if (g.ctl[MB_MODE] == 0)
        mb_push<NW>(g);
    else
        mb_pull<NW>(g);
}

// The last block to end the level advances it.  ctl is volatile there, other
// blocks' sums are not to come from this SM's cache.
template <int NW>
__global__ void __launch_bounds__(kMbThreads) k_mb_level_end(MbView g, int64_t cap, cudaGraphConditionalHandle h)
{
    if (g.ctl[MB_MODE] == 0)
        mb_push_end<NW>(g);
    else
        mb_pull_end<NW>(g);
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd((unsigned long long *)&g.ctl[MB_DONE], 1ull) != gridDim.x - 1) return;
    __threadfence();
    volatile int64_t *ctl = g.ctl;
    const int64_t nf = ctl[MB_NNEXT], fe = ctl[MB_FE_NEXT], nh = ctl[MB_NHUB_NEXT], cur = ctl[MB_CUR];
    const int64_t level = ctl[MB_LEVEL] + 1, levels = ctl[MB_LEVELS];
    ctl[MB_DONE] = 0;
    ctl[MB_NF] = nf;
    ctl[MB_NNEXT] = 0;
    ctl[MB_NHUB] = nh;
    ctl[MB_NHUB_NEXT] = 0;
    ctl[MB_FE] = fe;
    ctl[MB_FE_NEXT] = 0;
    ctl[MB_CUR] = cur ^ 1;
    ctl[MB_LEVEL] = level;
    if (level > levels) ctl[MB_LEVELS] = level;
    ctl[MB_MODE] = mb_mode(fe, g.nnz);
    cudaGraphSetConditional(h, (nf != 0 && level < cap) ? 1u : 0u);
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
    v.hubs0 = b.hubs[0];
    v.hubs1 = b.hubs[1];
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
    device_free(c, b.hubs[0]);
    device_free(c, b.hubs[1]);
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
    for (auto &hubs : b.hubs) GBC_TRY(device_alloc(ctx, (void **)&hubs, (g->nnz / kMbHub + 1) * sizeof(int32_t)));
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
            // resident blocks, and no more than have work
            auto grid = [&](const void *kernel, int64_t items) {
                return (int)std::min<int64_t>(occ_grid(ctx, kernel, kMbThreads, 0), items / kMbThreads + 1);
            };
            k_mb_level<NW><<<grid((const void *)k_mb_level<NW>, std::max((v.n + v.nitems) * NW, v.nnz)), kMbThreads, 0,
                             cs>>>(v);
            k_mb_level_end<NW><<<grid((const void *)k_mb_level_end<NW>, v.n * NW), kMbThreads, 0, cs>>>(v, v.n + 2, h);
            note_launches(2);
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
