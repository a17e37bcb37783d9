// Weakly connected components with min-id labels.
//
// Replaces wcc.c: min-label propagation over adjacency lists (wcc_algo,
// 30-42, with its pthread worklist 44-90) and over the grid and edge array
// (193-261), whose fixed point labels every vertex with the minimum vertex id
// of its component.
//
// GPU form: label propagation on component roots with pointer jumping.  Every
// edge hooks the larger of its two roots under the smaller one (atomicCAS on
// the root's parent word), so a root is always the minimum id of its tree;
// finds use path halving (pointer jumping), and a final pass jumps every
// vertex to its root.  The result equals the reference's fixed point bit for
// bit, independent of scheduling.
//
// With the adjacency built (after the sampling idea of Sutton et al.,
// "Optimizing parallel graph connectivity computation via subgraph sampling",
// IPDPS 2018):
//  1. every vertex takes the least of itself and its lists' first entries as
//     its parent (in-lists are in ascending order, so theirs is the least
//     in-neighbour): no atomics;
//  2. while the largest tree holds less than 7/8 of the sampled vertices, at
//     most EG_WCC_ROUNDS times: every tree's root is hooked under the least
//     root that the first four entries of its vertices' lists lead to (one
//     atomicMin per edge between trees, no finds), and the trees are flattened;
//  3. all entries of only those vertices that are not in the largest tree are
//     hooked with finds, which on power-law graphs skips most of the edges.
// The finds and hooks of two entries per list, in place of 1 and 2, were most
// of the time: undirected RMAT, 6,000,011 vertices 777 -> 201 us; undirected
// uniform, 3,000,011 vertices and 40 M entries 1.65 -> 0.8 ms.
#include <stdlib.h>

#include "eg_frontier.cuh"
#include "eg_internal.cuh"

#define EG_WCC_NONE 0xffffffffu

namespace {

__device__ __forceinline__ uint32_t uf_find(uint32_t *par, uint32_t x) {
    uint32_t p = __ldcg(par + x);
    while (p != x) {
        const uint32_t gp = __ldcg(par + p);
        if (gp != p) par[x] = gp;  // halve the path; parents only ever decrease
        x = p;
        p = gp;
    }
    return x;
}

__device__ __forceinline__ void uf_link(uint32_t *par, uint32_t x, uint32_t y) {
    uint32_t a = uf_find(par, x), b = uf_find(par, y);
    while (a != b) {
        if (a > b) {
            const uint32_t t = a;
            a = b;
            b = t;
        }
        const uint32_t old = atomicCAS(par + b, b, a);
        if (old == b) break;
        b = uf_find(par, old);
        a = uf_find(par, a);
    }
}

// The sampled largest tree (k_wcc_pick) and the hooks of the last round.
#define EG_WCC_ROUNDS 6
struct WccPick {
    uint32_t root, count, total, hooks;
};

// par[v] = the least of v and the first entries of its lists (optr NULL: one
// list); parents never exceed their children, so this is a forest.  Four
// vertices per thread, their loads in flight together.  bits: a bit per vertex
// with an edge.  Four vertices without one are done here: their root is
// written, their parent nowhere read, and the passes that follow leave them out
// by their bits (n = 16.8 M, 4 K entries: rest 61 us, flatten and labels 24 and
// 28 us with row pointers and parents read; a call 174 -> 107).
__global__ void __launch_bounds__(256) k_wcc_seed(const uint32_t *__restrict__ iptr, const uint32_t *__restrict__ icol,
                                                  const uint32_t *__restrict__ optr, const uint32_t *__restrict__ ocol,
                                                  uint32_t n, uint32_t *__restrict__ par,
                                                  uint32_t *__restrict__ root, uint32_t *__restrict__ bits) {
    const uint32_t nq = (uint32_t)(((uint64_t)n + 3) >> 2), lane = threadIdx.x & 31;
    // uniform trip count per warp
    for (uint32_t q0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); q0 < nq; q0 += gridDim.x * blockDim.x) {
        const uint32_t q = q0 + lane, v = 4 * q;
        uint32_t p[4] = {v, v + 1, v + 2, v + 3}, has = 0;
        for (int side = 0; side < 2 && q < nq; side++) {
            const uint32_t *__restrict__ ptr = side ? optr : iptr, *__restrict__ col = side ? ocol : icol;
            if (!ptr) break;
            const uint4 r = __ldg(reinterpret_cast<const uint4 *>(ptr + v));  // past the end: the buffer's padding
            const uint32_t b[5] = {r.x, r.y, r.z, r.w, __ldg(ptr + v + 4)};
            uint32_t c[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const bool on = v + i < n && b[i + 1] != b[i];
                c[i] = on ? __ldg(col + b[i]) : p[i];
                has |= (uint32_t)on << i;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) p[i] = c[i] < p[i] ? c[i] : p[i];
        }
        if (q < nq) reinterpret_cast<uint4 *>(has ? par : root)[q] = make_uint4(p[0], p[1], p[2], p[3]);
        uint32_t word = has << (4 * (lane & 7));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) word |= __shfl_xor_sync(EG_FULL_MASK, word, o);
        if (!(lane & 7) && q < nq) bits[q >> 3] = word;
    }
}
// Of the vertices 4 q .. 4 q + 3.
__device__ __forceinline__ bool wcc_any_edge(const uint32_t *__restrict__ bits, uint32_t q) {
    return (__ldg(bits + (q >> 3)) >> (4 * (q & 7))) & 15u;
}

// Roots of 512 sampled vertices with an edge (the first of four draws that
// has one), the most frequent one among them.  One CTA.
__global__ void __launch_bounds__(512) k_wcc_pick(const uint32_t *__restrict__ par, const uint32_t *__restrict__ iptr,
                                                   const uint32_t *__restrict__ optr, uint32_t n, WccPick *pick) {
    __shared__ __align__(16) uint32_t s_root[512];
    __shared__ unsigned long long s_best;
    uint32_t v[4], r = EG_WCC_NONE;
    bool has[4];
#pragma unroll
    for (uint32_t t = 0; t < 4; t++) {
        v[t] = (uint32_t)(((eg_mix64((uint64_t)threadIdx.x * 4 + t + 0x51ed) >> 32) * (uint64_t)n) >> 32);
        has[t] = iptr[v[t] + 1] != iptr[v[t]] || (optr && optr[v[t] + 1] != optr[v[t]]);
    }
    const uint32_t u = has[0] ? v[0] : has[1] ? v[1] : has[2] ? v[2] : v[3];
    if (has[0] | has[1] | has[2] | has[3]) r = par[u];
    s_root[threadIdx.x] = r;
    if (threadIdx.x == 0) s_best = 0;
    const uint32_t total = (uint32_t)__syncthreads_count(r != EG_WCC_NONE);
    uint32_t c = 0;
    for (uint32_t i = 0; i < 128; i++) {
        const uint4 x = reinterpret_cast<const uint4 *>(s_root)[i];
        c += (x.x == r) + (x.y == r) + (x.z == r) + (x.w == r);
    }
    if (r != EG_WCC_NONE) atomicMax(&s_best, ((unsigned long long)c << 32) | r);
    __syncthreads();
    if (threadIdx.x == 0) {
        pick->root = total ? (uint32_t)s_best : EG_WCC_NONE;
        pick->count = (uint32_t)(s_best >> 32);
        pick->total = total;
    }
}

// One round: root[] are the flattened roots, par[] is theirs on entry.
__global__ void __launch_bounds__(256) k_wcc_round(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ col,
                                                   const uint32_t *__restrict__ root,
                                                   const uint32_t *__restrict__ bits, uint32_t n, WccPick *pick,
                                                   uint32_t *par) {
    uint32_t hooks = 0;
    for (uint64_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
        if (!((__ldg(bits + (u >> 5)) >> (u & 31)) & 1u)) continue;
        const uint32_t ru = __ldg(root + u), b = __ldg(ptr + u), d = __ldg(ptr + u + 1) - b;
        uint32_t rw[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) rw[i] = i < d ? __ldg(col + b + i) : (uint32_t)u;
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) rw[i] = __ldg(root + rw[i]);
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const uint32_t lo = min(ru, rw[i]), hi = max(ru, rw[i]);
            if (lo != hi && __ldca(par + hi) > lo) hooks += atomicMin(par + hi, lo) == hi;
        }
    }
    hooks = __reduce_add_sync(EG_FULL_MASK, hooks);
    if (hooks && (threadIdx.x & 31) == 0) atomicAdd(&pick->hooks, hooks);
}

// Hooks the entries between trees of the vertices whose root was not the
// sampled tree's (root[]: the roots before this kernel): a warp walks the lists
// of 32 vertices together.  Entries inside a tree, nearly all by then, are told
// by root[]: with finds for every entry all vertices meet on the few words of
// the trees' roots (path of 1 M vertices through shuffled ids: 1046 us, now 27;
// mesh of 1000 x 1000 850, now 490).
__global__ void __launch_bounds__(256) k_wcc_rest(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ col,
                                                  const uint32_t *__restrict__ root,
                                                  const uint32_t *__restrict__ bits, uint32_t n,
                                                  const WccPick *__restrict__ pick, uint32_t *par) {
    const uint32_t skip = pick->root, lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint64_t v0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); v0 < n; v0 += stride) {
        const uint32_t u = (uint32_t)v0 + lane;
        const uint32_t on = __ldg(bits + (v0 >> 5));
        if (!on) continue;
        uint32_t b = 0, d = 0;
        if (((on >> lane) & 1u) && __ldg(root + u) != skip) {
            b = __ldg(ptr + u);
            d = __ldg(ptr + u + 1) - b;
        }
        if (!__any_sync(EG_FULL_MASK, d != 0u)) continue;
        eg_warp_lists(u, b, d, [&](bool valid, uint32_t, uint32_t ou, uint32_t p) {
            if (!valid) return;
            const uint32_t ru = __ldg(root + ou), rw = __ldg(root + __ldg(col + p));
            if (ru != rw) uf_link(par, ru, rw);
        });
    }
}

// The roots of vertices v .. v + 3 from their ancestors p.  The first
// EG_WCC_HOPS steps read the parents through L1 (the low ids are most vertices'
// ancestors; an old line holds an ancestor too).  Where they do not end, each
// step is written to the vertices' own parents and read past L1, so that the
// steps double: a forest of depth d takes EG_WCC_HOPS + log2(d) steps in place
// of d (ids in order along a path: the seeds make one chain of it).
#define EG_WCC_HOPS 6
__device__ __forceinline__ void wcc_roots(uint32_t *par, uint32_t n, uint32_t v, uint32_t (&p)[4]) {
    for (int hop = 0;; hop++) {  // parents only ever decrease: a stale one is still an ancestor
        uint32_t g[4];
        bool more = false;
#pragma unroll
        for (int i = 0; i < 4; i++) g[i] = hop < EG_WCC_HOPS ? __ldca(par + p[i]) : __ldcg(par + p[i]);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            more |= g[i] != p[i];
            p[i] = g[i];
        }
        if (!more) break;
        if (hop >= EG_WCC_HOPS) {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (v + i < n) __stcg(par + v + i, p[i]);
        }
    }
}

// Every vertex's root into par and root, four vertices per thread.
__global__ void __launch_bounds__(256) k_wcc_flatten(uint32_t n, uint32_t *par, uint32_t *__restrict__ root,
                                                     const uint32_t *__restrict__ bits) {
    const uint32_t nq = (uint32_t)(((uint64_t)n + 3) >> 2);
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        if (!wcc_any_edge(bits, q)) continue;
        const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(par) + q);
        const uint32_t v = 4 * q;
        uint32_t p[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (v + i >= n) p[i] = v;  // padding: any vertex
        wcc_roots(par, n, v, p);
        const uint4 y = make_uint4(p[0], p[1], p[2], p[3]);
        if (y.x != x.x || y.y != x.y || y.z != x.z || y.w != x.w) reinterpret_cast<uint4 *>(par)[q] = y;
        reinterpret_cast<uint4 *>(root)[q] = y;
    }
}

// Every vertex's label: its root.  With a pick, root[] holds the roots from
// before the last hooks: the vertices of the picked tree, mostly all, have
// one label between them, found once per thread.  Counts the components.
__global__ void __launch_bounds__(256) k_wcc_labels(uint32_t n, uint32_t *par, uint32_t *label,
                                                    const WccPick *pick, const uint32_t *__restrict__ bits,
                                                    unsigned long long *roots) {
    const uint32_t nq = (uint32_t)(((uint64_t)n + 3) >> 2);
    const uint32_t skip = pick ? pick->root : EG_WCC_NONE;
    uint32_t common = skip;
    if (skip != EG_WCC_NONE)
        for (uint32_t g; (g = __ldcg(par + common)) != common;) common = g;
    uint32_t count = 0;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        const uint32_t v = 4 * q;
        if (pick && !wcc_any_edge(bits, q)) {
            count += n - v < 4 ? n - v : 4;
            continue;
        }
        const uint4 x = __ldcg(reinterpret_cast<const uint4 *>(pick ? label : par) + q);
        uint32_t p[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (v + i >= n || p[i] == skip) p[i] = common;
            if (v + i >= n && skip == EG_WCC_NONE) p[i] = v;
        }
        if (p[0] != common || p[1] != common || p[2] != common || p[3] != common) wcc_roots(par, n, v, p);
#pragma unroll
        for (int i = 0; i < 4; i++) count += v + i < n && p[i] == v + i;
        if (!pick || p[0] != x.x || p[1] != x.y || p[2] != x.z || p[3] != x.w)
            reinterpret_cast<uint4 *>(label)[q] = make_uint4(p[0], p[1], p[2], p[3]);
    }
    count = __reduce_add_sync(EG_FULL_MASK, count);
    if ((threadIdx.x & 31) == 0 && count) atomicAdd(roots, (unsigned long long)count);
}

__global__ void k_wcc_init(uint32_t n, uint32_t *par) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) par[v] = v;
}

__global__ void k_wcc_hook(const uint32_t *__restrict__ pairs, uint64_t m, uint32_t *par, uint32_t *retries) {
    uint32_t tries = 0;
    for (uint64_t e = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; e < m; e += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 p = reinterpret_cast<const uint2 *>(pairs)[e];
        uint32_t a = uf_find(par, p.x), b = uf_find(par, p.y);
        while (a != b) {
            if (a > b) {
                uint32_t t = a;
                a = b;
                b = t;
            }
            // link root b (larger) under root a (smaller)
            const uint32_t old = atomicCAS(par + b, b, a);
            if (old == b) break;
            tries++;
            b = uf_find(par, old);
            a = uf_find(par, a);
        }
    }
    if (tries) atomicAdd(retries, tries);
}

__global__ void k_widen(const uint32_t *__restrict__ in, uint32_t n, long long *out) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) out[v] = in[v];
}

}  // namespace

extern "C" int eg_wcc(eg_graph *g, int64_t *labels_out, eg_wcc_stats *stats) {
    if (!g) return eg_fail(EG_EINVAL, "NULL graph");
    eg_ctx *ctx = g->ctx;
    EG_CUDA(cudaSetDevice(ctx->device));
    const uint32_t n = g->n;
    EG_TRY(eg_buf_ensure(ctx, g->label, (uint64_t)n * 4));  // padded: written four vertices at a time
    // work: parent[n] | counters | a bit per vertex | int64 staging for the host copy
    const uint64_t off_cnt = ((uint64_t)n + 3) & ~3ull, off_bits = off_cnt + 8;
    const uint64_t off_wide = off_bits + (((uint64_t)n + 127) / 128) * 4;
    EG_TRY(eg_buf_ensure(ctx, g->bfs_work, (off_wide + (labels_out ? 2ull * n : 0)) * 4));
    uint32_t *par = bp<uint32_t>(g->bfs_work);
    uint32_t *retries = par + off_cnt, *bits = par + off_bits;
    unsigned long long *roots = reinterpret_cast<unsigned long long *>(par + off_cnt + 2);
    long long *wide = reinterpret_cast<long long *>(par + off_wide);
    uint32_t blocks = (uint32_t)(ctx->sm_count * 8);
    EG_CUDA(cudaEventRecord(ctx->ev0, ctx->stream));
    EG_TRY(eg_zero(ctx, retries, 32, ctx->stream));
    const bool have_csr = (g->built & EG_LAYOUT_CSR) != 0;
    const bool sym = (g->flags & EG_UNDIRECTED) != 0;
    const bool have_csc = (g->built & EG_LAYOUT_CSC) != 0;
    int rounds = 1;
    const WccPick *picked = nullptr;
    if (have_csr && (sym || have_csc) && n >= 1024) {
        // an undirected graph's in- and out-lists hold the same neighbours
        const eg_adj &in = have_csc ? g->csc : g->csr;
        const uint32_t *iptr = bp<uint32_t>(in.ptr), *icol = bp<uint32_t>(in.col);
        const uint32_t *optr = sym ? nullptr : bp<uint32_t>(g->csr.ptr), *ocol = sym ? nullptr : bp<uint32_t>(g->csr.col);
        WccPick *pick = reinterpret_cast<WccPick *>(par + off_cnt + 4);
        uint32_t *root = bp<uint32_t>(g->label);
        k_wcc_seed<<<blocks, 256, 0, ctx->stream>>>(iptr, icol, optr, ocol, n, par, root, bits);
        EG_LAUNCHED(ctx);
        WccPick *hp = reinterpret_cast<WccPick *>(ctx->h_pinned);
        for (int r = 0;; r++) {
            k_wcc_flatten<<<blocks, 256, 0, ctx->stream>>>(n, par, root, bits);
            EG_LAUNCHED(ctx);
            k_wcc_pick<<<1, 512, 0, ctx->stream>>>(par, iptr, optr, n, pick);
            EG_LAUNCHED(ctx);
            EG_TRY(eg_readback_wait(ctx, hp, pick, sizeof(WccPick), ctx->stream));
            // most vertices in one tree, or a round that hooked next to nothing,
            // or entries so few that a round costs more than their finds
            if (r == EG_WCC_ROUNDS || 8ull * hp->count >= 7ull * hp->total || (r && hp->hooks < n / 256) ||
                g->m < n / 64)
                break;
            EG_TRY(eg_zero(ctx, &pick->hooks, 4, ctx->stream));
            k_wcc_round<<<blocks, 256, 0, ctx->stream>>>(iptr, icol, root, bits, n, pick, par);
            EG_LAUNCHED(ctx);
            if (!sym) {
                k_wcc_round<<<blocks, 256, 0, ctx->stream>>>(optr, ocol, root, bits, n, pick, par);
                EG_LAUNCHED(ctx);
            }
        }
        k_wcc_rest<<<blocks, 256, 0, ctx->stream>>>(iptr, icol, root, bits, n, pick, par);
        EG_LAUNCHED(ctx);
        if (!sym) {
            k_wcc_rest<<<blocks, 256, 0, ctx->stream>>>(optr, ocol, root, bits, n, pick, par);
            EG_LAUNCHED(ctx);
        }
        picked = pick;
        rounds = 2;
    } else {
        k_wcc_init<<<blocks, 256, 0, ctx->stream>>>(n, par);
        EG_LAUNCHED(ctx);
        if (g->m_in) {
            k_wcc_hook<<<blocks, 256, 0, ctx->stream>>>(bp<uint32_t>(g->pairs), g->m_in, par, retries);
            EG_LAUNCHED(ctx);
        }
    }
    k_wcc_labels<<<blocks, 256, 0, ctx->stream>>>(n, par, bp<uint32_t>(g->label), picked, bits, roots);
    EG_LAUNCHED(ctx);
    EG_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
    if (labels_out) {
        k_widen<<<blocks, 256, 0, ctx->stream>>>(bp<uint32_t>(g->label), n, wide);
        EG_LAUNCHED(ctx);
        EG_CUDA(cudaMemcpyAsync(labels_out, wide, (uint64_t)n * 8, cudaMemcpyDeviceToHost, ctx->stream));
    }
    unsigned long long *h = (unsigned long long *)ctx->h_pinned;
    EG_TRY(eg_readback_wait(ctx, h, roots, 8, ctx->stream));
    if (labels_out || stats) EG_CUDA(cudaStreamSynchronize(ctx->stream));
    if (stats) {
        stats->components = (uint32_t)*h;
        stats->rounds = rounds;
        EG_CUDA(cudaEventElapsedTime(&stats->ms, ctx->ev0, ctx->ev1));
    }
    return EG_OK;
}
