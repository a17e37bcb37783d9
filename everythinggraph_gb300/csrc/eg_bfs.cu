// Direction-optimising BFS with a bitmap frontier, and bit-sliced
// multi-source BFS.
//
// Replaces bfs_simple.c (bfs_push 121-134, bfs_pull 104-120, the switch rule
// 191-197) and bfsgrid_cilk.c (get_bfs 48-65, iterator 121-168).  The
// reference's frontier is a byte map plus id lists (random.c:74-77,
// buffer.c:62-297); here it is a bitmap in the style of Gemini's Bitmap
// (bitmap.h:16-50), plus a list with running edge sums for push levels.
//
// Levels follow the reference: level[root] = 1, unreached = 0 (the value
// bfsgrid_cilk and the edge-centric bfs_simple write into dist[]).
#include <stdlib.h>
#include <string.h>

#include "eg_bfsloop.cuh"
#include "eg_frontier.cuh"
#include "eg_internal.cuh"
#include "eg_mspull.cuh"

namespace {

#define EG_MS_STEP 4  // entries per lane in flight in the multi-source push

// first[v] = v's in-neighbour with the largest out-degree (the smallest id
// among equals), EG_NO_VERTEX when the in-list is empty: the in-neighbour
// most likely to be in a large frontier, checked before the list is read.
// One warp per vertex, 32 entries per step.
__global__ void k_first_in(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ col,
                           const uint32_t *__restrict__ deg, uint32_t n, uint32_t *__restrict__ first) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps) {
        const uint32_t b = ptr[v], e = ptr[v + 1];
        unsigned long long best = 0ull;  // (degree << 32) | ~id: the max is the largest degree, then the smallest id
        for (uint64_t p = (uint64_t)b + lane; p < e; p += 32) {  // p + 32 may not fit 32 bits
            const uint32_t u = col[p];
            const unsigned long long key = ((unsigned long long)deg[u] << 32) | (uint32_t)~u;
            best = key > best ? key : best;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long y = __shfl_down_sync(EG_FULL_MASK, best, o);
            best = y > best ? y : best;
        }
        if (lane == 0) first[v] = b < e ? ~(uint32_t)best : EG_NO_VERTEX;
    }
}

// bits[w]: bit l set when vertex 32w + l has no in-neighbours (ids past n: set)
__global__ void k_no_in_bits(const uint32_t *__restrict__ first, uint32_t n, uint32_t nw, uint32_t *bits) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;  // a multiple of 32: warps stay whole
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < (uint64_t)nw * 32; v += stride) {
        const bool none = v >= n || first[v] == EG_NO_VERTEX;
        const uint32_t b = __ballot_sync(EG_FULL_MASK, none);
        if ((threadIdx.x & 31) == 0) bits[v >> 5] = b;
    }
}

}  // namespace

extern "C" void eg_bfs_opts_default(eg_bfs_opts *o) {
    if (!o) return;
    o->direction = EG_BFS_AUTO;
    o->switch_divisor = -1.0;
    o->device_parents = 0;
    o->host_loop = -1;
}

static uint32_t blocks_for(eg_ctx *ctx, uint64_t threads) {
    uint64_t b = (threads + 255) / 256;
    uint64_t cap = (uint64_t)ctx->sm_count * 8;
    if (b > cap) b = cap;
    return b ? (uint32_t)b : 1u;
}

// first_in: one word per vertex, padded to whole 16-byte reads, then the bits of
// the vertices without in-neighbours
static uint64_t first_words(uint32_t n) { return ((uint64_t)n + 3) & ~3ull; }

static int bfs_check(eg_graph *g, const eg_bfs_opts *opts, eg_bfs_opts &o) {
    if (!g) return eg_fail(EG_EINVAL, "NULL graph");
    if (!(g->built & EG_LAYOUT_CSR)) return eg_fail(EG_ENOTBUILT, "BFS needs the CSR");
    if (opts) o = *opts;
    else eg_bfs_opts_default(&o);
    if (o.direction < EG_BFS_AUTO || o.direction > EG_BFS_PULL_ONLY) return eg_fail(EG_EINVAL, "bad direction");
    return EG_OK;
}

// One BFS from `root` into the device arrays of output slot `slot` (g->level
// / g->parent, or g->level_s / g->parent_s), on the context stream.  When
// level_out / parent_out are given, the copies to them are queued before the
// final wait; returns once the traversal (and those copies) are done.
static int bfs_core(eg_graph *g, uint32_t root, const eg_bfs_opts &o, int slot, bool want_parent, int32_t *level_out,
                    int32_t *parent_out, eg_bfs_stats *stats) {
    if (root >= g->n) return eg_fail(EG_EINVAL, "root %u >= n %u", root, g->n);
    const bool undirected = (g->flags & EG_UNDIRECTED) != 0;
    // in-lists: the CSC when built (sorted by source id, so RMAT hubs come first
    // and bottom-up scans stop early); an undirected CSR is its own transpose
    eg_adj *in_adj = (g->built & EG_LAYOUT_CSC) ? &g->csc : (undirected ? &g->csr : nullptr);
    if (!in_adj && o.direction != EG_BFS_PUSH_ONLY)
        return eg_fail(EG_ENOTBUILT, "bottom-up BFS on a directed graph needs the CSC");
    eg_ctx *ctx = g->ctx;
    EG_CUDA(cudaSetDevice(ctx->device));
    const uint32_t n = g->n;
    const uint32_t nw = (n + 31) >> 5;
    if (in_adj && g->first_in_src != in_adj->col.p) {  // once per graph and in-list array
        // first_in[0 .. n), then the bit per vertex without in-neighbours
        EG_TRY(eg_buf_ensure(ctx, g->first_in, (first_words(n) + nw) * 4));
        k_first_in<<<(uint32_t)ctx->sm_count * 8, 256, 0, ctx->stream>>>(
            bp<uint32_t>(in_adj->ptr), bp<uint32_t>(in_adj->col), bp<uint32_t>(g->out_deg), n, bp<uint32_t>(g->first_in));
        EG_LAUNCHED(ctx);
        k_no_in_bits<<<blocks_for(ctx, (uint64_t)nw * 32), 256, 0, ctx->stream>>>(bp<uint32_t>(g->first_in), n, nw,
                                                                                  bp<uint32_t>(g->first_in) + first_words(n));
        EG_LAUNCHED(ctx);
        g->first_in_src = in_adj->col.p;
    }
    eg_buf &lbuf = slot ? g->level_s[slot - 1] : g->level, &pbuf = slot ? g->parent_s[slot - 1] : g->parent;
    EG_TRY(eg_buf_ensure(ctx, lbuf, (uint64_t)n * 4));
    if (want_parent) EG_TRY(eg_buf_ensure(ctx, pbuf, (uint64_t)n * 4));
    // work: list [n uint4] | visited | prev | bm0 | bm1 | state
    const uint64_t nw4 = ((uint64_t)nw + 3) & ~3ull, off_vis = 4ull * n, off_st = (off_vis + 4 * nw4 + 7) & ~7ull;
    EG_TRY(eg_buf_ensure(ctx, g->bfs_work, (off_st + sizeof(BfsLoopState) / 4) * 4));
    uint32_t *wk = bp<uint32_t>(g->bfs_work), *bits = wk + off_vis;
    BfsLoopState *st = reinterpret_cast<BfsLoopState *>(wk + off_st);
    int32_t *level = bp<int32_t>(lbuf);
    int32_t *parent = want_parent ? bp<int32_t>(pbuf) : nullptr;
    const double divisor = o.switch_divisor < 0 ? g->bfs_divisor : o.switch_divisor;
    const double threshold = divisor > 0 ? (double)g->m / divisor : 0.0;
    const unsigned long long whole = threshold < 0x1p40 ? (unsigned long long)threshold : 1ull << 40;
    const uint32_t *first = in_adj ? bp<uint32_t>(g->first_in) : nullptr;
    BfsLoop a{bp<uint32_t>(g->csr.ptr), bp<uint32_t>(g->csr.col), in_adj ? bp<uint32_t>(in_adj->ptr) : nullptr,
              in_adj ? bp<uint32_t>(in_adj->col) : nullptr, first, first ? first + first_words(n) : nullptr,
              bp<uint32_t>(g->out_deg), n, nw, root, o.direction, threshold, whole, level, parent,
              bits, bits + nw4, {bits + 2 * nw4, bits + 3 * nw4}, reinterpret_cast<uint4 *>(wk), st};
    const uint64_t want = (g->m + n) / EG_BFSL_SHARE + 1, most = (uint64_t)ctx->sm_count * EG_BFSL_B;
    void *args[] = {&a};
    EG_CUDA(cudaEventRecord(ctx->ev0, ctx->stream));
    EG_CUDA(cudaLaunchCooperativeKernel(parent ? (const void *)k_bfs_loop<true> : (const void *)k_bfs_loop<false>,
                                        dim3((uint32_t)(want < most ? want : most)), dim3(EG_BFSL_T), args, 0, ctx->stream));
    ctx->launches++;
    EG_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
    if (level_out) EG_CUDA(cudaMemcpyAsync(level_out, level, (uint64_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    if (parent_out) EG_CUDA(cudaMemcpyAsync(parent_out, parent, (uint64_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    BfsLoopState *h = reinterpret_cast<BfsLoopState *>(ctx->h_pinned);
    EG_TRY(eg_readback_wait(ctx, h, st, sizeof(BfsLoopState), ctx->stream));
    if (h->err) return eg_fail(EG_ETIMEOUT, "BFS did not terminate");
    if (stats) {
        stats->levels = (int)h->levels;
        stats->reached = (uint32_t)h->reached;
        stats->edges_traversed = h->traversed;
        stats->pull_levels = (int)h->pull_levels;
        EG_CUDA(cudaEventSynchronize(ctx->ev1));  // the flag may be seen before the event's completion
        EG_CUDA(cudaEventElapsedTime(&stats->ms, ctx->ev0, ctx->ev1));
    }
    return EG_OK;
}

extern "C" int eg_bfs(eg_graph *g, uint32_t root, const eg_bfs_opts *opts, int32_t *level_out, int32_t *parent_out,
                      eg_bfs_stats *stats) {
    eg_bfs_opts o;
    EG_TRY(bfs_check(g, opts, o));
    EG_CUDA(cudaSetDevice(g->ctx->device));
    return bfs_core(g, root, o, 0, parent_out != nullptr || o.device_parents, level_out, parent_out, stats);
}

// BFS from each root in turn; root i's levels (and parents) go to
// level_out + i * n (parent_out + i * n).  Root i is traversed into output
// slot i % EG_OUT_SLOTS and copied out on the copy stream while the next
// roots are traversed into the other slots; a slot is rewritten only after
// its previous copy-out.
extern "C" int eg_bfs_batch(eg_graph *g, const uint32_t *roots, uint32_t k, const eg_bfs_opts *opts,
                            int32_t *level_out, int32_t *parent_out, eg_bfs_stats *stats) {
    eg_bfs_opts o;
    EG_TRY(bfs_check(g, opts, o));
    if (!roots && k) return eg_fail(EG_EINVAL, "NULL roots");
    for (uint32_t i = 0; i < k; i++)
        if (roots[i] >= g->n) return eg_fail(EG_EINVAL, "root %u >= n %u", roots[i], g->n);
    eg_ctx *ctx = g->ctx;
    EG_CUDA(cudaSetDevice(ctx->device));
    const uint64_t n = g->n;
    const bool want_parent = parent_out != nullptr || o.device_parents;
    int rc = EG_OK;
    for (uint32_t i = 0; i < k && rc == EG_OK; i++) {
        const int slot = (int)(i % EG_OUT_SLOTS);
        if (i >= EG_OUT_SLOTS) EG_CUDA(cudaStreamWaitEvent(ctx->stream, ctx->ev_out[EG_OUT_SLOTS + slot], 0));
        rc = bfs_core(g, roots[i], o, slot, want_parent, nullptr, nullptr, stats ? stats + i : nullptr);
        if (rc != EG_OK) break;
        if (level_out || parent_out) {
            const int32_t *level = bp<int32_t>(slot ? g->level_s[slot - 1] : g->level);
            const int32_t *parent = want_parent ? bp<int32_t>(slot ? g->parent_s[slot - 1] : g->parent) : nullptr;
            EG_CUDA(cudaEventRecord(ctx->ev_out[slot], ctx->stream));
            EG_CUDA(cudaStreamWaitEvent(ctx->copy_stream, ctx->ev_out[slot], 0));
            if (level_out)
                EG_CUDA(cudaMemcpyAsync(level_out + i * n, level, n * 4, cudaMemcpyDeviceToHost, ctx->copy_stream));
            if (parent_out)
                EG_CUDA(cudaMemcpyAsync(parent_out + i * n, parent, n * 4, cudaMemcpyDeviceToHost, ctx->copy_stream));
            EG_CUDA(cudaEventRecord(ctx->ev_out[EG_OUT_SLOTS + slot], ctx->copy_stream));
        }
    }
    const cudaError_t e = cudaStreamSynchronize(ctx->copy_stream);
    if (rc == EG_OK && e != cudaSuccess) return eg_fail(EG_ECUDA, "BFS batch copies: %s", cudaGetErrorString(e));
    return rc;
}

// ============================================================== multi-source
// Bit-sliced BFS: bit s of seen[v] / front[v] belongs to source s (k <= 64).
namespace {
struct MsCounters {
    unsigned long long deg;   // sum of out-degrees of vertices with a nonzero new word
    unsigned long long tdeg;  // sum over new (vertex, source) pairs of the vertex's out-degree
    unsigned long long disc;  // new (vertex, source) pairs
    unsigned long long sel;   // push: vertices listed by k_ms_queue << 32 | their entries
    uint32_t count;           // vertices with a nonzero new word
    uint32_t nheavy;          // pull: k_msp_mid's list
    uint32_t nhuge;           // pull: k_msp_heavy's list
};

__global__ void k_ms_init(uint32_t n, unsigned long long *seen, unsigned long long *front) {
    uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
        seen[v] = 0ull;
        front[v] = 0ull;
    }
}

// Device state of the multi-source level loop (one CUDA graph, see
// msbfs_graph_build): the frontier's size and out-degree sum, the direction
// chosen for the level, and the totals for the stats.
struct MsGState {
    uint32_t count;  // vertices in the frontier
    int32_t lvl;     // level of the frontier (roots: 1)
    int pull;        // this level runs bottom-up
    int pull_levels;
    unsigned long long fdeg;       // out-degree sum of the frontier's vertices
    unsigned long long reached;    // (vertex, source) pairs reached
    unsigned long long traversed;  // sum over those pairs of the vertex's out-degree
    unsigned long long m;          // adjacency entries (switch rule)
    uint32_t n;
    uint32_t pad;
};

// Roots: seen/front bits, level 1, and the first frontier (distinct roots)
// with its statistics.  One block of 64 threads.
__global__ void k_ms_roots(const uint32_t *roots, int k, uint32_t n, unsigned long long *seen, unsigned long long *front,
                           int32_t *levels, const uint32_t *__restrict__ deg, MsGState *st, unsigned long long m) {
    __shared__ unsigned int s_count;
    __shared__ unsigned long long s_fdeg, s_rdeg;
    const int s = threadIdx.x;
    if (s == 0) {
        s_count = 0;
        s_fdeg = 0;
        s_rdeg = 0;
    }
    __syncthreads();
    if (s < k) {
        const uint32_t r = roots[s];
        atomicOr(seen + r, 1ull << s);
        const unsigned long long was = atomicOr(front + r, 1ull << s);
        if (levels) levels[(uint64_t)s * n + r] = 1;
        const unsigned long long d = deg[r];
        atomicAdd(&s_rdeg, d);
        if (!was) {  // the first source at this vertex counts it
            atomicAdd(&s_count, 1u);
            atomicAdd(&s_fdeg, d);
        }
    }
    __syncthreads();
    if (s == 0) {
        st->count = s_count;
        st->lvl = 1;
        st->pull = 0;
        st->pull_levels = 0;
        st->fdeg = s_fdeg;
        st->reached = (unsigned long long)k;
        st->traversed = s_rdeg;
        st->m = m;
        st->n = n;
    }
}

// Level start: the reference's switch rule (bfs_simple.c:191-197) on the
// frontier's size and out-degrees, and cleared level counters.
__global__ void k_msg_prep(MsGState *st, MsCounters *cnt) {
    st->pull = (double)st->count + (double)st->fdeg > (double)st->m / 20.0;
    cnt->deg = 0;
    cnt->tdeg = 0;
    cnt->disc = 0;
    cnt->count = 0;
    cnt->sel = 0;
    cnt->nheavy = 0;
    cnt->nhuge = 0;
}

// Push levels: lists the vertices with a nonzero frontier word and out-edges
// as (running sum of their entries, first entry - that sum, vertex); four
// vertices per thread, one atomic per 1024 vertices.
__global__ void __launch_bounds__(256) k_ms_queue(uint32_t n, const unsigned long long *__restrict__ front,
                                                  const uint32_t *__restrict__ ptr, uint4 *queue, const MsGState *st,
                                                  MsCounters *cnt) {
    __shared__ unsigned long long s_warp[8], s_base;
    if (st->pull) return;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t b0 = blockIdx.x * 1024ull; b0 < n; b0 += gridDim.x * 1024ull) {
        const uint64_t v0 = b0 + 4 * threadIdx.x;
        const uint32_t v = (uint32_t)v0;
        uint32_t bits = 0, r[5];
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (v0 + i < n && front[v0 + i] != 0ull) bits |= 1u << i;
        bfsl_rows(ptr, v, bits != 0u, r);
        unsigned long long mine = 0;  // vertices << 32 | entries (m < 2^32)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (r[i + 1] == r[i]) bits &= ~(1u << i);
            if ((bits >> i) & 1u) mine += (1ull << 32) | (r[i + 1] - r[i]);
        }
        unsigned long long x = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(EG_FULL_MASK, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long t = 0;
            for (int w = 0; w < 8; w++) {
                const unsigned long long y = s_warp[w];
                s_warp[w] = t;
                t += y;
            }
            s_base = t ? atomicAdd(&cnt->sel, t) : 0ull;
        }
        __syncthreads();
        const unsigned long long at = s_base + s_warp[warp] + x - mine;
        uint32_t pos = (uint32_t)(at >> 32), off = (uint32_t)at;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (!((bits >> i) & 1u)) continue;
            queue[pos++] = make_uint4(off, r[i] - off, v + i, 0u);
            off += r[i + 1] - r[i];
        }
        __syncthreads();  // s_warp and s_base are rewritten for the next 1024
    }
}

// Push: every warp takes an equal share of the listed vertices' entries, hubs
// included (eg_frontier.cuh's list), and hands each entry's vertex the sources
// that it lacks.  Words read through L1 may be old: the atomicOr settles it.
// Bound by its chain of loads and the launches around it.  (A warp walked 32
// vertices' lists, the ones over 256 entries by chunks in two launches more:
// list and push took 101 us of a 64-source batch on undirected RMAT n = 2^20,
// now 41; of a 32-source one on n = 1.7K, m = 45K 88, now 29.)
__global__ void __launch_bounds__(256) k_ms_push(const uint32_t *__restrict__ col, const uint4 *__restrict__ queue,
                                                 const MsGState *st, const unsigned long long *__restrict__ seen,
                                                 const unsigned long long *__restrict__ front,
                                                 unsigned long long *next, const MsCounters *cnt) {
    if (st->pull) return;
    const uint32_t qlen = (uint32_t)(cnt->sel >> 32), E = (uint32_t)cnt->sel;
    const uint32_t lane = threadIdx.x & 31, le = eg_lanemask_lt() | (1u << lane);
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t per = (uint32_t)(((uint64_t)E + warps - 1) / warps);
    per = per < 64u ? 64u : (per + 31u) & ~31u;
    const uint64_t begin = (uint64_t)wid * per;
    if (begin >= E) return;
    uint32_t p = (uint32_t)begin;
    const uint32_t end = E - p > per ? p + per : E;
    uint32_t i0 = eg_list_find(&queue[0].x, 4u, qlen, p);
    for (; p < end; i0 += 32) {
        uint4 q = make_uint4(0xffffffffu, 0u, 0u, 0u);
        unsigned long long f = 0ull;
        if (i0 + lane < qlen) {
            q = __ldg(queue + i0 + lane);
            f = __ldg(front + q.z);
        }
        const uint32_t wend = i0 + 32 < qlen ? __ldg(&queue[i0 + 32].x) : E;
        const uint32_t stop = wend < end ? wend : end;
        for (; p < stop; p = stop - p > 32 * EG_MS_STEP ? p + 32 * EG_MS_STEP : stop) {
            uint32_t v[EG_MS_STEP];
            unsigned long long add[EG_MS_STEP], was[EG_MS_STEP];
            bool on[EG_MS_STEP];
#pragma unroll
            for (int k = 0; k < EG_MS_STEP; k++) {
                const uint32_t x0 = p + 32 * k;
                const uint32_t starts = __reduce_or_sync(EG_FULL_MASK, q.x - x0 < 32u ? 1u << (q.x - x0) : 0u);
                const uint32_t o = __popc(__ballot_sync(EG_FULL_MASK, q.x < x0)) - 1 + __popc(starts & le);
                const uint32_t at = x0 + lane + __shfl_sync(EG_FULL_MASK, q.y, o);
                add[k] = __shfl_sync(EG_FULL_MASK, f, o);
                on[k] = stop - p > 32u * k + lane;
                v[k] = on[k] ? __ldg(col + at) : 0u;
            }
#pragma unroll
            for (int k = 0; k < EG_MS_STEP; k++) {
                was[k] = on[k] ? __ldca(next + v[k]) : ~0ull;
                add[k] &= on[k] ? ~__ldg(seen + v[k]) : 0ull;
            }
#pragma unroll
            for (int k = 0; k < EG_MS_STEP; k++)
                if (add[k] & ~was[k]) atomicOr(next + v[k], add[k]);
        }
    }
}

// Level end: the new frontier's counters into the loop state; the while node
// repeats the level body while the frontier is non-empty (and at most n + 1
// levels, a bound the loop can never need).
__global__ void k_msg_end(MsGState *st, const MsCounters *cnt, cudaGraphConditionalHandle handle) {
    st->count = cnt->count;
    st->fdeg = cnt->deg;
    st->reached += cnt->disc;
    st->traversed += cnt->tdeg;
    st->pull_levels += st->pull;
    st->lvl += 1;
    cudaGraphSetConditional(handle, (cnt->count > 0 && (uint32_t)st->lvl <= st->n + 1) ? 1u : 0u);
}

// Folds the new words into seen, records levels, makes them the frontier and
// counts it.  The warp writes the levels source by source (a row of levels is
// one source's), so that a store covers up to 32 consecutive words; every
// lane walking its own word's sources wrote 32 rows at once, and four
// atomics per warp met on the counters (64 sources, undirected RMAT-20:
// 694 us in 7 levels, now 220).
__global__ void __launch_bounds__(256) k_ms_fold(uint32_t n, unsigned long long *seen, unsigned long long *front,
                                                 unsigned long long *next, int32_t *levels, const MsGState *st,
                                                 const uint32_t *__restrict__ deg, MsCounters *cnt) {
    const int32_t lvl = st->lvl + 1;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t stride = gridDim.x * blockDim.x;
    unsigned long long sum[3] = {0ull, 0ull, 0ull};  // out-degrees, out-degrees per new pair, new pairs
    uint32_t count = 0;
    // uniform trip count per warp for the collectives
    for (uint64_t v0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); v0 < n; v0 += stride) {
        const uint64_t v = v0 + lane;
        unsigned long long x = 0ull;
        if (v < n) {
            x = next[v];
            if (x) {
                next[v] = 0ull;
                const unsigned long long s = seen[v];
                x &= ~s;
                if (x) seen[v] = s | x;
            }
            front[v] = x;
        }
        if (!__any_sync(EG_FULL_MASK, x != 0ull)) continue;
        if (x) {
            const unsigned long long d = deg[v], pc = (unsigned long long)__popcll((long long)x);
            sum[0] += d;
            sum[1] += d * pc;
            sum[2] += pc;
            count++;
        }
        if (levels) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t mine = (uint32_t)(x >> (32 * h));
                uint32_t any = __reduce_or_sync(EG_FULL_MASK, mine);
                while (any) {
                    const uint32_t s = (uint32_t)__ffs(any) - 1;
                    any &= any - 1;
                    if ((mine >> s) & 1u) levels[(uint64_t)(32 * h + s) * n + v] = lvl;
                }
            }
        }
    }
    __shared__ unsigned long long s_sum[8][3];
    __shared__ uint32_t s_cnt[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        count += __shfl_down_sync(EG_FULL_MASK, count, o);
#pragma unroll
        for (int i = 0; i < 3; i++) sum[i] += __shfl_down_sync(EG_FULL_MASK, sum[i], o);
    }
    if (lane == 0) {
        s_cnt[warp] = count;
        for (int i = 0; i < 3; i++) s_sum[warp][i] = sum[i];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) {
            count += s_cnt[w];
            for (int i = 0; i < 3; i++) sum[i] += s_sum[w][i];
        }
        if (count) {
            atomicAdd(&cnt->count, count);
            atomicAdd(&cnt->deg, sum[0]);
            atomicAdd(&cnt->tdeg, sum[1]);
            atomicAdd(&cnt->disc, sum[2]);
        }
    }
}
}  // namespace

// The level loop of eg_bfs_multi as one CUDA graph: a while node whose body
// is prep (direction), the push (list, entries) or the three-part pull, fold,
// and end (counters into the state, loop condition).  Valid while the
// buffers and k it was captured with (key) stay the same.
static int msbfs_graph_build(eg_graph *g, const void *const key[8], const eg_adj *in_adj,
                             unsigned long long all, unsigned long long *seen, unsigned long long *front,
                             unsigned long long *next, uint4 *queue, int32_t *levels,
                             MsGState *st, MsCounters *cnt) {
    eg_ctx *ctx = g->ctx;
    eg_bfs_graph &bg = g->msg;
    const uint32_t n = g->n;
    const uint32_t *deg = bp<uint32_t>(g->out_deg);
    if (bg.exec) cudaGraphExecDestroy(bg.exec);
    if (bg.graph) cudaGraphDestroy(bg.graph);
    bg.exec = nullptr;
    bg.graph = nullptr;
    cudaGraph_t graph = nullptr;
    EG_CUDA(cudaGraphCreate(&graph, 0));
    bg.graph = graph;
    cudaGraphConditionalHandle handle;
    EG_CUDA(cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t wnode;
    EG_CUDA(cudaGraphAddNode(&wnode, graph, nullptr, nullptr, 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    const uint32_t blocks = (uint32_t)ctx->sm_count * 8;
    EG_CUDA(cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    k_msg_prep<<<1, 1, 0, ctx->stream>>>(st, cnt);
    k_ms_queue<<<blocks, 256, 0, ctx->stream>>>(n, front, bp<uint32_t>(g->csr.ptr), queue, st, cnt);
    k_ms_push<<<blocks, 256, 0, ctx->stream>>>(bp<uint32_t>(g->csr.col), queue, st, seen, front, next, cnt);
    // the pull's lists share the push's (idle in a pull level)
    uint32_t *heavy = reinterpret_cast<uint32_t *>(queue), *huge = heavy + n;
    k_msp_light<<<blocks, 256, 0, ctx->stream>>>(bp<uint32_t>(in_adj->ptr), bp<uint32_t>(in_adj->col), n, all, seen,
                                                 front, next, heavy, &cnt->nheavy, &st->pull);
    k_msp_mid<<<blocks, 256, 0, ctx->stream>>>(bp<uint32_t>(in_adj->ptr), bp<uint32_t>(in_adj->col), all, seen, front,
                                               next, heavy, &cnt->nheavy, huge, &cnt->nhuge, &st->pull);
    k_msp_heavy<<<blocks, 256, 0, ctx->stream>>>(bp<uint32_t>(in_adj->ptr), bp<uint32_t>(in_adj->col), all, seen, front,
                                                 next, huge, &cnt->nhuge, &st->pull);
    k_ms_fold<<<blocks, 256, 0, ctx->stream>>>(n, seen, front, next, levels, st, deg, cnt);
    k_msg_end<<<1, 1, 0, ctx->stream>>>(st, cnt, handle);
    cudaError_t ce = cudaStreamEndCapture(ctx->stream, &body);
    if (ce != cudaSuccess) return eg_fail(EG_ECUDA, "multi-source BFS capture: %s", cudaGetErrorString(ce));
    cudaGraphExec_t exec = nullptr;
    EG_TRY(eg_graph_instantiate(ctx, &exec, graph));
    bg.exec = exec;
    for (int i = 0; i < 8; i++) bg.key[i] = key[i];
    return EG_OK;
}

extern "C" int eg_bfs_multi(eg_graph *g, const uint32_t *roots, int k, int32_t *levels_out, eg_bfs_stats *stats) {
    if (!g || !roots) return eg_fail(EG_EINVAL, "NULL argument");
    if (k < 1 || k > 64) return eg_fail(EG_EINVAL, "k=%d sources: bit-sliced BFS takes 1..64", k);
    if (!(g->built & EG_LAYOUT_CSR)) return eg_fail(EG_ENOTBUILT, "BFS needs the CSR");
    const bool undirected = (g->flags & EG_UNDIRECTED) != 0;
    // in-lists: the CSC when built (sorted by source id, so RMAT hubs come first
    // and bottom-up scans stop early); an undirected CSR is its own transpose
    eg_adj *in_adj = (g->built & EG_LAYOUT_CSC) ? &g->csc : (undirected ? &g->csr : nullptr);
    if (!in_adj) return eg_fail(EG_ENOTBUILT, "multi-source BFS on a directed graph needs the CSC");
    for (int s = 0; s < k; s++)
        if (roots[s] >= g->n) return eg_fail(EG_EINVAL, "root %u >= n", roots[s]);
    eg_ctx *ctx = g->ctx;
    EG_CUDA(cudaSetDevice(ctx->device));
    const uint32_t n = g->n;
    // work: push list (uint4) | seen | front | next (u64 each) | roots | counters | state
    EG_TRY(eg_buf_ensure(ctx, g->msbfs_work, 40ull * n + 64 * 4 + 64 + 64));
    uint4 *queue = bp<uint4>(g->msbfs_work);
    unsigned long long *seen = reinterpret_cast<unsigned long long *>(queue + n);
    unsigned long long *front = seen + n, *next = seen + 2ull * n;
    uint32_t *d_roots = reinterpret_cast<uint32_t *>(seen + 3ull * n);
    MsCounters *cnt = reinterpret_cast<MsCounters *>(d_roots + 64);
    MsGState *st = reinterpret_cast<MsGState *>(d_roots + 64 + 16);
    int32_t *levels = nullptr;
    if (levels_out) {
        EG_TRY(eg_buf_ensure(ctx, g->level, (uint64_t)k * n * 4));
        levels = bp<int32_t>(g->level);
    }
    const uint32_t *deg = bp<uint32_t>(g->out_deg);
    const unsigned long long all = k == 64 ? ~0ull : ((1ull << k) - 1ull);
    const void *key[8] = {g->msbfs_work.p, levels, g->csr.col.p, in_adj->col.p, (const void *)(uintptr_t)k, g->csr.ptr.p,
                          in_adj->ptr.p, g->out_deg.p};
    bool same = g->msg.exec != nullptr;
    for (int i = 0; i < 8 && same; i++) same = g->msg.key[i] == key[i];
    if (!same)
        EG_TRY(msbfs_graph_build(g, key, in_adj, all, seen, front, next, queue, levels, st, cnt));
    EG_CUDA(cudaMemcpyAsync(d_roots, roots, (uint64_t)k * 4, cudaMemcpyHostToDevice, ctx->stream));
    EG_CUDA(cudaEventRecord(ctx->ev0, ctx->stream));
    if (levels) EG_CUDA(cudaMemsetAsync(levels, 0, (uint64_t)k * n * 4, ctx->stream));
    k_ms_init<<<blocks_for(ctx, n), 256, 0, ctx->stream>>>(n, seen, front);
    EG_LAUNCHED(ctx);
    EG_CUDA(cudaMemsetAsync(next, 0, (uint64_t)n * 8, ctx->stream));
    k_ms_roots<<<1, 64, 0, ctx->stream>>>(d_roots, k, n, seen, front, levels, deg, st, g->m);
    EG_LAUNCHED(ctx);
    EG_CUDA(cudaGraphLaunch(g->msg.exec, ctx->stream));
    ctx->launches++;
    EG_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
    MsGState *h = (MsGState *)ctx->h_pinned;
    EG_CUDA(cudaMemcpyAsync(h, st, sizeof(MsGState), cudaMemcpyDeviceToHost, ctx->stream));
    if (levels_out) EG_CUDA(cudaMemcpyAsync(levels_out, levels, (uint64_t)k * n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    EG_CUDA(cudaStreamSynchronize(ctx->stream));
    if ((uint32_t)h->lvl > n + 1) return eg_fail(EG_ETIMEOUT, "multi-source BFS did not terminate");
    if (stats) {
        stats->levels = h->lvl - 1;
        stats->reached = (uint32_t)(h->reached > 0xffffffffull ? 0xffffffffull : h->reached);
        stats->edges_traversed = h->traversed;
        stats->pull_levels = h->pull_levels;
        EG_CUDA(cudaEventElapsedTime(&stats->ms, ctx->ev0, ctx->ev1));
    }
    return EG_OK;
}

int eg_bfs_tune(eg_graph *g, float *ms, double *divisor) {
    // per-root times vary several-fold (an early switch to pull costs a few
    // roots a lot), so the mean is taken over 48 sampled roots
    static const double kDiv[5] = {20.0, 40.0, 80.0, 160.0, 320.0};
    constexpr int R = 48;
    uint32_t roots[R];
    EG_TRY(eg_sample_roots(g, R, 12345, roots));
    for (int d = 0; d < 5; d++) {
        eg_bfs_opts o;
        eg_bfs_opts_default(&o);
        o.switch_divisor = kDiv[d];
        o.device_parents = 1;
        eg_bfs_stats st;
        EG_TRY(eg_bfs(g, roots[0], &o, nullptr, nullptr, &st));  // warm-up (buffers)
        float t = 0.f;
        for (int r = 0; r < R; r++) {
            EG_TRY(eg_bfs(g, roots[r], &o, nullptr, nullptr, &st));
            t += st.ms / (float)R;
        }
        if (d == 0 || t < *ms) {
            *ms = t;
            *divisor = kDiv[d];
        }
    }
    g->bfs_divisor = *divisor;
    return EG_OK;
}
