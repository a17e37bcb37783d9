// Batched personalised PageRank: up to 32 queries advance together, one
// warp lane per query.
//
// No reference counterpart (the reference runs one global PageRank); the
// per-query iteration is pr_numa's correct pull PR (pr_numa.c:245-277,396)
// with the teleport and dangling mass sent to the query's seed set:
//   x'[v] = d * sum_{u->v} x[u]/deg[u] + (1 - d + d * dangling(x)) * t[v]
// where t is uniform over the query's seeds.  Each query stops when the FP64
// L1 change of its vector drops below its tolerance or after max_iters.
//
// Layout: vertex-major [n][32] fp32 rows (128 bytes per vertex), so for an
// entry u->v a group of 8 lanes reads x[u][0..31] with one 16-byte load each.
// The rows are summed from a work list made once per graph (eg_ppr_plan):
// rows in order of length, the long ones in parts whose sums are added in
// part order.  A lane only ever combines its own queries' values, in an order
// fixed by the graph, so each query's result is bit-identical whether it runs
// alone or in a batch.
#include <stdlib.h>
#include <string.h>

#include "eg_ppr.cuh"


namespace {
// Sweep-loop state of the batched PageRank graph.
struct PprLoop {
    int sweeps;
    int max_sweeps;
    int nq;
    int pad;
};

__global__ void k_ppr_loop_init(PprLoop *st, int max_sweeps, int nq) {
    st->sweeps = 0;
    st->max_sweeps = max_sweeps;
    st->nq = nq;
}

// Sweep end: the while node runs another sweep while a query of the batch is
// still running (and fewer than max_iters sweeps ran).
__global__ void k_ppr_loop_end(PprLoop *st, const PprQ *qs, cudaGraphConditionalHandle handle) {
    st->sweeps += 1;
    bool all = true;
    for (int q = 0; q < st->nq; q++) all &= qs[q].done != 0;
    cudaGraphSetConditional(handle, (!all && st->sweeps < st->max_sweeps) ? 1u : 0u);
}

// The sweep loop of eg_ppr_multi as one CUDA graph: a while node whose body
// is one sweep (row sums of the 32 lanes, the sums of rows in parts, seeds'
// teleport, finish and the per-query FP64 reductions) and the
// loop test.  Valid while the buffers, nq and the
// options it was captured with (key) stay the same.
int ppr_graph_build(eg_graph *g, const void *const key[8], uint32_t fin_blocks, const eg_ppr_opts &o, int nq, float *R,
                    float *X, float *Y, float *psum, double2 *part, const uint32_t *d_seeds, const uint32_t *d_soff, PprQ *qs, PprLoop *lst) {
    eg_ctx *ctx = g->ctx;
    eg_bfs_graph &bg = g->ppg;
    if (bg.exec) cudaGraphExecDestroy(bg.exec);
    if (bg.graph) cudaGraphDestroy(bg.graph);
    bg.exec = nullptr;
    bg.graph = nullptr;
    const uint32_t n = g->n;
    const uint32_t *deg = bp<uint32_t>(g->out_deg);
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
    EG_CUDA(cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    if (g->ppr_nlong + g->ppr_nrows)
        k_ppr_rows<<<(uint32_t)ctx->sm_count * EG_PPR_MINB, 256, 0, ctx->stream>>>(
            bp<uint32_t>(g->csc.ptr), bp<uint32_t>(g->csc.col), bp<uint4>(g->ppr_long), g->ppr_nlong,
            bp<uint32_t>(g->ppr_order), g->ppr_nrows, X, Y, psum);
    if (g->ppr_nmulti)
        k_ppr_fixup<<<eg_div_up((uint64_t)g->ppr_nmulti * 32, 256), 256, 0, ctx->stream>>>(
            bp<uint4>(g->ppr_multi), g->ppr_nmulti, psum, Y);
    k_ppr_seeds<<<1, EG_PPR_LANES, 0, ctx->stream>>>(d_seeds, d_soff, d_soff + 1, nq, qs, o.damping, Y,
                                                     bp<uint32_t>(g->csc.ptr));
    k_ppr_finish<<<fin_blocks, 256, 0, ctx->stream>>>(Y, deg, n, o.damping, qs, R, X, part);
    k_ppr_reduce<<<EG_PPR_LANES, 128, 0, ctx->stream>>>(part, fin_blocks, qs, 1);
    k_ppr_loop_end<<<1, 1, 0, ctx->stream>>>(lst, qs, handle);
    cudaError_t ce = cudaStreamEndCapture(ctx->stream, &body);
    if (ce != cudaSuccess) return eg_fail(EG_ECUDA, "batched PageRank capture: %s", cudaGetErrorString(ce));
    cudaGraphExec_t exec = nullptr;
    EG_TRY(eg_graph_instantiate(ctx, &exec, graph));
    bg.exec = exec;
    for (int i = 0; i < 8; i++) bg.key[i] = key[i];
    return EG_OK;
}

// Vertex v's in-list: a whole row's key orders it by length, longest first
// (EG_PPR_PART - 1 - entries), rows without entries and long rows last; a
// long row reserves its parts, counts[0] of them, and a place in `multi`,
// counts[1] of them.  counts[2]: the whole rows with entries.
__global__ void __launch_bounds__(256) k_ppr_plan_rows(const uint32_t *__restrict__ ptr, uint32_t n, uint32_t *keys,
                                                       uint32_t *vals, uint4 *multi, uint32_t *counts) {
    uint32_t whole = 0;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const uint32_t len = ptr[v + 1] - ptr[v];
        const bool fits = len && len < EG_PPR_PART;
        keys[v] = fits ? EG_PPR_PART - 1 - len : EG_PPR_PART - 1;
        vals[v] = v;
        whole += fits;
        if (len >= EG_PPR_PART) {
            const uint32_t parts = (len - 1) / EG_PPR_PART + 1;
            multi[atomicAdd(counts + 1, 1u)] = make_uint4(v, atomicAdd(counts, parts), parts, 0u);
        }
    }
    whole = __reduce_add_sync(EG_FULL_MASK, whole);
    if ((threadIdx.x & 31) == 0 && whole) atomicAdd(counts + 2, whole);
}
// A warp per long row: its parts' items.
__global__ void __launch_bounds__(256) k_ppr_plan_parts(const uint32_t *__restrict__ ptr,
                                                        const uint4 *__restrict__ multi, uint32_t nmulti,
                                                        uint4 *__restrict__ longs) {
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= nmulti) return;
    const uint4 r = multi[t];
    const uint32_t b = ptr[r.x], e = ptr[r.x + 1];
    for (uint32_t k = lane; k < r.z; k += 32) {
        const uint32_t at = b + k * EG_PPR_PART;
        longs[r.y + k] = make_uint4(at, min(EG_PPR_PART, e - at), r.y + k, 0u);
    }
}
}  // namespace

int eg_ppr_plan(eg_graph *g) {
    if (g->ppr_planned) return EG_OK;
    eg_ctx *ctx = g->ctx;
    const uint32_t n = g->n;
    // at most m / EG_PPR_PART rows are long, and 2 m / EG_PPR_PART parts are theirs
    const uint64_t most = g->m / EG_PPR_PART;
    eg_buf kb, vb, ko;
    int rc = EG_OK;
    auto cleanup = [&]() {
        cudaStreamSynchronize(ctx->stream);
        for (eg_buf *b : {&kb, &vb, &ko}) eg_buf_free(ctx, *b);
    };
#define QTRY(x)            \
    do {                   \
        rc = (x);          \
        if (rc != EG_OK) { \
            cleanup();     \
            return rc;     \
        }                  \
    } while (0)
    QTRY(eg_buf_ensure(ctx, kb, (uint64_t)n * 4 + 16));
    QTRY(eg_buf_ensure(ctx, vb, (uint64_t)n * 4));
    QTRY(eg_buf_ensure(ctx, ko, (uint64_t)n * 4));
    QTRY(eg_buf_ensure(ctx, g->ppr_order, (uint64_t)n * 4));
    QTRY(eg_buf_ensure(ctx, g->ppr_multi, most * sizeof(uint4) + 16));
    uint32_t *counts = bp<uint32_t>(kb) + n;
    const uint32_t blocks = (uint32_t)ctx->sm_count * 8;
    QTRY(eg_zero(ctx, counts, 12, ctx->stream));
    k_ppr_plan_rows<<<blocks, 256, 0, ctx->stream>>>(bp<uint32_t>(g->csc.ptr), n, bp<uint32_t>(kb), bp<uint32_t>(vb),
                                                     bp<uint4>(g->ppr_multi), counts);
    ctx->launches++;
    uint32_t *h = (uint32_t *)ctx->h_pinned;
    QTRY(eg_readback_wait(ctx, h, counts, 12, ctx->stream));
    const uint32_t nlong = h[0], nmulti = h[1], nrows = h[2];
    uint32_t *ks, *vs;
    QTRY(eg_radix_sort(ctx, bp<uint32_t>(kb), bp<uint32_t>(vb), bp<uint32_t>(ko), bp<uint32_t>(g->ppr_order), n, 9, &ks,
                       &vs));
    if (vs != bp<uint32_t>(g->ppr_order) &&  // one vertex: nothing was sorted
        cudaMemcpyAsync(g->ppr_order.p, vs, (uint64_t)n * 4, cudaMemcpyDeviceToDevice, ctx->stream) != cudaSuccess)
        QTRY(eg_fail(EG_ECUDA, "personalised PageRank plan"));
    QTRY(eg_buf_ensure(ctx, g->ppr_long, (uint64_t)nlong * sizeof(uint4) + 16));
    if (nmulti) {
        k_ppr_plan_parts<<<eg_div_up((uint64_t)nmulti * 32, 256), 256, 0, ctx->stream>>>(
            bp<uint32_t>(g->csc.ptr), bp<uint4>(g->ppr_multi), nmulti, bp<uint4>(g->ppr_long));
        ctx->launches++;
    }
    if (cudaStreamSynchronize(ctx->stream) != cudaSuccess)
        QTRY(eg_fail(EG_ECUDA, "personalised PageRank plan: %s", cudaGetErrorString(cudaGetLastError())));
#undef QTRY
    cleanup();
    // a captured sweep holds the last plan's buffers and counts
    eg_bfs_graph &bg = g->ppg;
    if (bg.exec) cudaGraphExecDestroy(bg.exec);
    if (bg.graph) cudaGraphDestroy(bg.graph);
    bg = eg_bfs_graph();
    g->ppr_nlong = nlong;
    g->ppr_nmulti = nmulti;
    g->ppr_nrows = nrows;
    g->ppr_planned = true;
    return EG_OK;
}

extern "C" int eg_ppr_multi(eg_graph *g, const uint32_t *seeds, const uint32_t *seed_offsets, int nq,
                            const eg_ppr_opts *opts, float *ranks_out, eg_ppr_stats *stats) {
    if (!g || !seeds || !seed_offsets) return eg_fail(EG_EINVAL, "NULL argument");
    if (nq < 1 || nq > EG_PPR_LANES) return eg_fail(EG_EINVAL, "nq=%d: a batch holds 1..32 queries", nq);
    if (!(g->built & EG_LAYOUT_CSC) || !(g->built & EG_LAYOUT_CSR))
        return eg_fail(EG_ENOTBUILT, "personalised PageRank needs the CSC and the out-degrees");
    eg_ppr_opts o;
    if (opts) o = *opts;
    else {
        o.damping = 0.85f;
        o.max_iters = 50;
        for (int q = 0; q < EG_PPR_LANES; q++) o.tolerance[q] = 1e-6f;
    }
    if (o.max_iters < 1 || !(o.damping > 0.f && o.damping < 1.f)) return eg_fail(EG_EINVAL, "bad PPR options");
    const uint32_t n = g->n;
    for (int q = 0; q < nq; q++) {
        if (seed_offsets[q + 1] <= seed_offsets[q]) return eg_fail(EG_EINVAL, "query %d has no seed", q);
        for (uint32_t i = seed_offsets[q]; i < seed_offsets[q + 1]; i++)
            if (seeds[i] >= n) return eg_fail(EG_EINVAL, "seed %u >= n", seeds[i]);
    }
    eg_ctx *ctx = g->ctx;
    EG_CUDA(cudaSetDevice(ctx->device));
    EG_TRY(eg_ppr_plan(g));
    const uint32_t nseeds_total = seed_offsets[nq];
    const uint32_t fin_blocks = (uint32_t)ctx->sm_count * 4;
    // work: R, X, Y [n*32 f32] | part sums [nlong*32 f32] | block partials | seeds | offsets | queries
    const uint64_t vec = (uint64_t)n * EG_PPR_LANES;
    const uint64_t off_X = vec, off_Y = 2 * vec, off_ps = 3 * vec,
                   off_part = off_ps + (uint64_t)g->ppr_nlong * EG_PPR_LANES,
                   off_seeds = off_part + (uint64_t)fin_blocks * 32 * 4,
                   off_soff = off_seeds + nseeds_total + 8, off_q = (off_soff + 40 + 63) & ~63ull,
                   off_loop = off_q + 32 * sizeof(PprQ) / 4;
    EG_TRY(eg_buf_ensure(ctx, g->ppr_work, (off_loop + 64) * 4));
    float *W = bp<float>(g->ppr_work);
    float *R = W, *X = W + off_X, *Y = W + off_Y, *psum = W + off_ps;
    double2 *part = reinterpret_cast<double2 *>(W + off_part);
    uint32_t *d_seeds = reinterpret_cast<uint32_t *>(W + off_seeds);
    uint32_t *d_soff = reinterpret_cast<uint32_t *>(W + off_soff);
    PprQ *qs = reinterpret_cast<PprQ *>(W + off_q);
    PprLoop *lst = reinterpret_cast<PprLoop *>(W + off_loop);
    PprQ hq[EG_PPR_LANES];
    memset(hq, 0, sizeof(hq));
    for (int q = 0; q < nq; q++) {
        hq[q].active = 1;
        hq[q].tol = o.tolerance[q];
        hq[q].max_iters = o.max_iters;
        hq[q].nseeds = (int)(seed_offsets[q + 1] - seed_offsets[q]);
    }
    const uint32_t *deg = bp<uint32_t>(g->out_deg);
    EG_CUDA(cudaMemcpyAsync(d_seeds, seeds, (uint64_t)nseeds_total * 4, cudaMemcpyHostToDevice, ctx->stream));
    EG_CUDA(cudaMemcpyAsync(d_soff, seed_offsets, ((uint64_t)nq + 1) * 4, cudaMemcpyHostToDevice, ctx->stream));
    EG_CUDA(cudaMemcpyAsync(qs, hq, sizeof(hq), cudaMemcpyHostToDevice, ctx->stream));
    EG_CUDA(cudaEventRecord(ctx->ev0, ctx->stream));
    const uint32_t lanes = nq == 32 ? 0xffffffffu : ((1u << nq) - 1u);
    k_ppr_init<<<(uint32_t)ctx->sm_count * 8, 256, 0, ctx->stream>>>(n, 0xffffffffu, R, X);
    EG_LAUNCHED(ctx);
    k_ppr_empty<<<(uint32_t)ctx->sm_count * 8, 256, 0, ctx->stream>>>(bp<uint32_t>(g->csc.ptr), n, Y);
    EG_LAUNCHED(ctx);
    k_ppr_init_seeds<<<1, EG_PPR_LANES, 0, ctx->stream>>>(d_seeds, d_soff, d_soff + 1, lanes, qs, deg, R, X);
    EG_LAUNCHED(ctx);
    k_ppr_init_dangling<<<1, EG_PPR_LANES, 0, ctx->stream>>>(d_seeds, d_soff, d_soff + 1, lanes, deg, R, qs);
    EG_LAUNCHED(ctx);
    PprQ *hqs = (PprQ *)ctx->h_pinned;
    // the sweeps: one CUDA graph launch (a while node over one sweep)
    k_ppr_loop_init<<<1, 1, 0, ctx->stream>>>(lst, o.max_iters, nq);
    EG_LAUNCHED(ctx);
    uint32_t dmg;
    memcpy(&dmg, &o.damping, 4);
    // n and m are the graph's own, a new plan drops the capture; the seed
    // offsets' place follows the seed count
    const void *key[8] = {W, g->csc.col.p, nullptr, (const void *)(uintptr_t)nq, (const void *)(uintptr_t)dmg, d_soff,
                          g->csc.ptr.p, g->out_deg.p};
    eg_bfs_graph &bg = g->ppg;
    bool same = bg.exec != nullptr;
    for (int i = 0; i < 8 && same; i++) same = bg.key[i] == key[i];
    if (!same)
        EG_TRY(ppr_graph_build(g, key, fin_blocks, o, nq, R, X, Y, psum, part, d_seeds, d_soff, qs, lst));
    EG_CUDA(cudaGraphLaunch(bg.exec, ctx->stream));
    ctx->launches += 1;
    PprLoop *hl = reinterpret_cast<PprLoop *>(hqs + EG_PPR_LANES);
    EG_TRY(eg_readback(ctx, hl, lst, sizeof(PprLoop), ctx->stream));
    EG_CUDA(cudaStreamSynchronize(ctx->stream));
    const int it = hl->sweeps;
    EG_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
    if (ranks_out) {  // Y is free after the last sweep: the rows go through it
        k_ppr_extract<<<(uint32_t)ctx->sm_count * 8, 256, 0, ctx->stream>>>(R, n, nq, Y);
        EG_LAUNCHED(ctx);
        EG_CUDA(cudaMemcpyAsync(ranks_out, Y, (uint64_t)nq * n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    }
    EG_CUDA(cudaMemcpyAsync(hqs, qs, sizeof(PprQ) * EG_PPR_LANES, cudaMemcpyDeviceToHost, ctx->stream));
    EG_CUDA(cudaStreamSynchronize(ctx->stream));
    if (stats) {
        for (int q = 0; q < nq; q++) {
            stats->iterations[q] = hqs[q].iters;
            stats->residual[q] = hqs[q].residual;
        }
        stats->sweeps = it;
        EG_CUDA(cudaEventElapsedTime(&stats->ms, ctx->ev0, ctx->ev1));
    }
    return EG_OK;
}
