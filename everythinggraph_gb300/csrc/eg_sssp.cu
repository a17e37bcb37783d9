// Single- and multi-source SSSP: relaxation rounds with atomicMin, ordered by
// distance.
//
// Replaces sssp_pushpull.c: the push relax (sssp_algo, 39-56, which the
// reference runs with unit weights) and the weighted pull relax
// (sssp_algo_pull, 69-98) iterated to a fixed point (iterator, 127-190).  The
// fixed point is the exact shortest-path distance, which is what both this
// code and the reference's pull-only run (-a 1 -r) produce.  dist[root] = 0,
// unreached = UINT32_MAX-1 (sssp_pushpull.c:8).
//
// Weights are computed from the edge's endpoints, like the reference's
// CREATE_WEIGHT path (init_all.c:661-686), once per rule, and kept in CSR order.
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

#include "eg_frontier.cuh"
#include "eg_internal.cuh"

namespace {

using WRule = eg_wrule;

// ---- one source
// Label-correcting search in rounds, ordered by work.  A vertex whose distance
// dropped is active (one bit); a round relaxes the out-lists of the active
// vertices of least distance, as many distance buckets of them as make up
// EG_SSSP_MIN_WORK edges or 1 / EG_SSSP_PART of the active vertices' edges, whichever
// is more, and leaves the others active.  Relaxing every active vertex at once
// (frontier Bellman-Ford) scans each list again whenever a shorter path shows
// up: 3.4 scans of every edge on RMAT-20 with weights 1..255 in 13 rounds,
// against 1.1 to 1.2 in 16 to 20 here; buckets of a fixed width need 50 rounds
// for 1.4 scans (a CPU count of the rounds).  Any order ends in the same least
// fixed point, and a round holds the active vertex of least distance, which is
// final: at most n rounds.  Directed RMAT-23, weights 1..255: 5.5 -> 1.8 ms.
//
// A round is three kernels in the body of a CUDA-graph while node:
//   k_sssp_hist    edges of the active vertices per distance bucket; the last
//                  CTA picks the last bucket of the round and sets the loop
//                  condition
//   k_sssp_select  lists the round's vertices with the running sum of their
//                  list lengths, and clears their bits
//   k_sssp_push    the listed edges in equal shares per warp
// Directed RMAT-23 (weights 1..255) with EG_SSSP_MIN_WORK 2^20 /
// 2^21 / 2^22: 33 / 26 / 22 rounds, 2.31 / 1.98 / 1.80 ms; EG_SSSP_PART 8 / 16 /
// 32 / 64: 1.78 / 1.75 / 1.35 / 1.35 scans per edge (buckets of 1/64 of the
// largest weight; 1/128: 1.08, 1/256: 1.06 with a slower histogram).
#define EG_SSSP_BUCKETS 1024u
#define EG_SSSP_WBITS 7   // 2^7 buckets to the largest weight
#define EG_SSSP_PART 32u
#define EG_SSSP_MIN_WORK (1u << 22)
struct SsspState {
    unsigned long long sel;    // this round's list: vertices << 32 | edges
    unsigned long long relax;  // edges listed so far
    uint32_t base;             // no active distance is below this (in the rule's encoding)
    uint32_t low;              // least active distance seen by this round's histogram
    uint32_t last;             // last bucket of the round
    uint32_t done;             // CTAs of the histogram that are finished
    uint32_t rounds, limit, err, pad;
    uint32_t hist[EG_SSSP_BUCKETS];
};

// Buckets of an active distance: 2^shift units (u32 rules), 2^-7 (fp32, weights up to 1).
struct SsspBuckets {
    int f32;
    uint32_t shift;
    __device__ __forceinline__ uint32_t of(uint32_t d, uint32_t base) const {
        const uint32_t b = f32 ? (uint32_t)fminf((__uint_as_float(d) - __uint_as_float(base)) * 128.f, 1e6f)
                               : (d - base) >> shift;
        return b < EG_SSSP_BUCKETS ? b : EG_SSSP_BUCKETS - 1;
    }
    // no distance past bucket b of `base` is below this
    __device__ __forceinline__ uint32_t end(uint32_t base, uint32_t b, uint32_t inf) const {
        if (f32) return min(__float_as_uint(__uint_as_float(base) + (float)(b + 1) * 0.0078125f), inf);
        const uint64_t x = (uint64_t)base + ((uint64_t)(b + 1) << shift);
        return x < inf ? (uint32_t)x : inf;
    }
};

// The first bucket at which the running sum reaches the round's work, in a
// CTA of 256 threads, four buckets per thread (c: the thread's running sums,
// c[3] = sum): the last one when all of it is within min_work.  Returns the
// total; every thread gets `last`.
__device__ __forceinline__ unsigned long long sssp_pick(const unsigned long long (&c)[4], unsigned long long sum,
                                                        unsigned long long min_work, unsigned long long *s_sum,
                                                        uint32_t *s_last, uint32_t *last) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(EG_FULL_MASK, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_sum[warp] = x;
    __syncthreads();
    if (threadIdx.x == 0) *s_last = EG_SSSP_BUCKETS - 1;
    __syncthreads();
    unsigned long long before = x - sum, total = 0;
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) {
        if (i < warp) before += s_sum[i];
        total += s_sum[i];
    }
    if (total > min_work) {
        const unsigned long long part = total / EG_SSSP_PART;
        const unsigned long long want = part > min_work ? part : min_work;
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (before + c[i] >= want && before + (i ? c[i - 1] : 0ull) < want) *s_last = threadIdx.x * 4 + i;
    }
    __syncthreads();
    *last = *s_last;
    return total;
}

__global__ void k_sssp_init(uint32_t n, uint32_t nw, uint32_t *dist, uint32_t root, uint32_t *bm, SsspState *st,
                            uint32_t inf, uint32_t limit) {
    const uint32_t stride = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
    for (uint32_t v = i0; v < n; v += stride) dist[v] = v == root ? 0u : inf;
    for (uint32_t w = i0; w < nw; w += stride) bm[w] = w == root >> 5 ? 1u << (root & 31) : 0u;
    if (i0 < EG_SSSP_BUCKETS) st->hist[i0] = 0;
    if (i0 == 0) {
        st->sel = st->relax = 0;
        st->base = 0;
        st->low = 0xffffffffu;
        st->last = 0;
        st->done = 0;
        st->rounds = 0;
        st->limit = limit;
        st->err = 0;
    }
}

// Warps take 32 bitmap words at a time, one per lane, then walk them four
// together: f(g, v, bits) for group g of 0 .. 7 that has a set bit, lane l
// holding vertices v .. v + 3 (v a multiple of 4: one 16-byte load per array)
// and their 4 bits.  Walking them one vertex per lane took three times the
// instructions, which bounded the passes over a dense active set.
template <class F>
__device__ __forceinline__ void sssp_groups(uint32_t w0, uint32_t word, F &&f) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t some = __ballot_sync(EG_FULL_MASK, word != 0u);
#pragma unroll 1
    for (uint32_t g = 0; g < 8; g++) {
        if (!((some >> (4 * g)) & 15u)) continue;
        const uint32_t bits = (__shfl_sync(EG_FULL_MASK, word, 4 * g + (lane >> 3)) >> (4 * (lane & 7))) & 15u;
        f(g, (w0 + 4 * g) * 32 + 4 * lane, bits);
    }
}
// Row starts ptr[v .. v + 4] (past the end: the buffers' padding).
__device__ __forceinline__ void sssp_rows(const uint32_t *__restrict__ ptr, uint32_t v, bool on, uint32_t (&r)[5]) {
    const uint4 q = on ? __ldg(reinterpret_cast<const uint4 *>(ptr + v)) : make_uint4(0u, 0u, 0u, 0u);
    r[0] = q.x;
    r[1] = q.y;
    r[2] = q.z;
    r[3] = q.w;
    r[4] = on ? __ldg(ptr + v + 4) : 0u;
}
__device__ __forceinline__ void sssp_dists(const uint32_t *__restrict__ dist, uint32_t v, bool on, uint32_t (&d)[4]) {
    const uint4 q = on ? __ldg(reinterpret_cast<const uint4 *>(dist + v)) : make_uint4(0u, 0u, 0u, 0u);
    d[0] = q.x;
    d[1] = q.y;
    d[2] = q.z;
    d[3] = q.w;
}

// Groups of 4 words whose rows and distances are in flight, and CTAs per SM
// (each adds its buckets to the shared ones).  Passes of a directed RMAT search,
// n = 8.4M / n = 300K: 1 group, 8 CTAs 377 / 164 us; 2, 8 508 / 163; 4, 8 427 /
// 144; 4, 4 334 / 143; 4, 2 431 / 144.
#define EG_SSSP_HSTEP 4u
#define EG_SSSP_HB 4u
__global__ void __launch_bounds__(256) k_sssp_hist(const uint32_t *__restrict__ bm, uint32_t nw,
                                                   const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ dist,
                                                   SsspBuckets bk, SsspState *st, cudaGraphConditionalHandle handle) {
    __shared__ uint32_t s_hist[EG_SSSP_BUCKETS];
    __shared__ uint32_t s_low, s_last;
    __shared__ unsigned long long s_sum[8];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < EG_SSSP_BUCKETS; i += 256) s_hist[i] = 0;
    if (threadIdx.x == 0) s_low = 0xffffffffu;
    __syncthreads();
    const uint32_t base = st->base;
    uint32_t low = 0xffffffffu;
    for (uint32_t w0 = (blockIdx.x * 8 + warp) * 32; w0 < nw; w0 += gridDim.x * 256) {
        const uint32_t word = w0 + lane < nw ? __ldg(bm + w0 + lane) : 0u;
        const uint32_t some = __ballot_sync(EG_FULL_MASK, word != 0u);
#pragma unroll 1
        for (uint32_t g = 0; g < 8; g += EG_SSSP_HSTEP) {
            if (!((some >> (4 * g)) & ((1ull << (4 * EG_SSSP_HSTEP)) - 1))) continue;
            uint32_t r[EG_SSSP_HSTEP][5], d[EG_SSSP_HSTEP][4], bits[EG_SSSP_HSTEP];
#pragma unroll
            for (uint32_t j = 0; j < EG_SSSP_HSTEP; j++) {
                bits[j] = (__shfl_sync(EG_FULL_MASK, word, 4 * (g + j) + (lane >> 3)) >> (4 * (lane & 7))) & 15u;
                const uint32_t v = (w0 + 4 * (g + j)) * 32 + 4 * lane;
                sssp_rows(ptr, v, bits[j] != 0u, r[j]);
                sssp_dists(dist, v, bits[j] != 0u, d[j]);
            }
#pragma unroll
            for (uint32_t j = 0; j < EG_SSSP_HSTEP; j++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (!((bits[j] >> i) & 1u)) continue;
                    low = d[j][i] < low ? d[j][i] : low;
                    if (r[j][i + 1] != r[j][i]) atomicAdd(&s_hist[bk.of(d[j][i], base)], r[j][i + 1] - r[j][i]);
                }
        }
    }
    low = __reduce_min_sync(EG_FULL_MASK, low);
    if (lane == 0 && low != 0xffffffffu) atomicMin(&s_low, low);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < EG_SSSP_BUCKETS; i += 256)
        if (s_hist[i]) atomicAdd(&st->hist[i], s_hist[i]);
    if (threadIdx.x == 0) {
        if (s_low != 0xffffffffu) atomicMin(&st->low, s_low);
        __threadfence();
    }
    __syncthreads();  // every thread's adds are out before the CTA counts as done
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // the last CTA: four buckets per thread, their running sum
    unsigned long long c[4], sum = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        c[i] = sum += __ldcg(&st->hist[threadIdx.x * 4 + i]);
        st->hist[threadIdx.x * 4 + i] = 0;
    }
    uint32_t last;
    const unsigned long long total = sssp_pick(c, sum, EG_SSSP_MIN_WORK, s_sum, &s_last, &last);
    if (threadIdx.x == 0) {
        st->last = last;
        st->done = 0;
        st->sel = 0;
        if (total) st->rounds += 1;
        const bool over = total && st->rounds > st->limit;
        if (over) st->err = 1;
        cudaGraphSetConditional(handle, total && !over ? 1u : 0u);
    }
}

// List entry: x = first place of its list among the round's edges, y = what
// to add to a place to get the CSR entry, z = the vertex's distance.
__global__ void __launch_bounds__(256) k_sssp_select(uint32_t *__restrict__ bm, uint32_t nw,
                                                     const uint32_t *__restrict__ ptr,
                                                     const uint32_t *__restrict__ dist, SsspBuckets bk, SsspState *st,
                                                     uint4 *__restrict__ queue) {
    __shared__ uint32_t s_cnt[8], s_edges[8];
    __shared__ unsigned long long s_base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t base = st->base, last = st->last;
    // uniform trip count per CTA
    for (uint32_t c0 = blockIdx.x * 256; c0 < nw; c0 += gridDim.x * 256) {
        const uint32_t w0 = c0 + warp * 32;
        const uint32_t word = w0 + lane < nw ? bm[w0 + lane] : 0u;
        uint32_t keep = 0;                // bits 4g .. 4g + 3: the lane's listed vertices of group g
        uint32_t g_cnt = 0, g_edges = 0;  // of group `lane`
        sssp_groups(w0, word, [&](uint32_t g, uint32_t v, uint32_t bits) {
            uint32_t r[5], d[4];
            sssp_rows(ptr, v, bits != 0u, r);
            sssp_dists(dist, v, bits != 0u, d);
            uint32_t clear = 0, k = 0, e = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (((bits >> i) & 1u) && bk.of(d[i], base) <= last) {
                    clear |= 1u << i;
                    if (r[i + 1] != r[i]) k |= 1u << i;
                    e += r[i + 1] - r[i];
                }
            }
            keep |= k << (4 * g);
            const uint32_t c = __reduce_add_sync(EG_FULL_MASK, __popc(k));
            e = __reduce_add_sync(EG_FULL_MASK, e);
            if (lane == g) {
                g_cnt = c;
                g_edges = e;
            }
            // the words without the listed bits: eight lanes hold a word's
            uint32_t left = (bits & ~clear) << (4 * (lane & 7)), any = clear;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                left |= __shfl_xor_sync(EG_FULL_MASK, left, o);
                any |= __shfl_xor_sync(EG_FULL_MASK, any, o);
            }
            if (!(lane & 7) && any) bm[w0 + 4 * g + (lane >> 3)] = left;
        });
        uint32_t xc = g_cnt, xe = g_edges;  // inclusive scans over the groups (lanes 0 .. 7)
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const uint32_t yc = __shfl_up_sync(EG_FULL_MASK, xc, o), ye = __shfl_up_sync(EG_FULL_MASK, xe, o);
            if (lane >= (uint32_t)o) {
                xc += yc;
                xe += ye;
            }
        }
        if (lane == 7) {
            s_cnt[warp] = xc;
            s_edges[warp] = xe;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t tc = 0, te = 0;
            for (int i = 0; i < 8; i++) {
                const uint32_t a = s_cnt[i], b = s_edges[i];
                s_cnt[i] = tc;
                s_edges[i] = te;
                tc += a;
                te += b;
            }
            // both sums in one word (a round lists at most m < 2^32 edges),
            // so that places and edges keep the same order
            s_base = tc ? atomicAdd(&st->sel, ((unsigned long long)tc << 32) | te) : 0ull;
        }
        __syncthreads();
        const uint32_t pc = (uint32_t)(s_base >> 32) + s_cnt[warp] + xc - g_cnt;
        const uint32_t pe = (uint32_t)s_base + s_edges[warp] + xe - g_edges;
        if (__any_sync(EG_FULL_MASK, keep != 0u)) {
#pragma unroll 1
            for (uint32_t g = 0; g < 8; g++) {
                const uint32_t bits = (keep >> (4 * g)) & 15u;
                if (!__any_sync(EG_FULL_MASK, bits != 0u)) continue;
                const uint32_t v = (w0 + 4 * g) * 32 + 4 * lane;
                uint32_t r[5], d[4];
                sssp_rows(ptr, v, bits != 0u, r);
                sssp_dists(dist, v, bits != 0u, d);
                uint32_t len = 0;
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if ((bits >> i) & 1u) len += r[i + 1] - r[i];
                uint32_t xl = len, xk = __popc(bits);
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t yl = __shfl_up_sync(EG_FULL_MASK, xl, o), yk = __shfl_up_sync(EG_FULL_MASK, xk, o);
                    if (lane >= (uint32_t)o) {
                        xl += yl;
                        xk += yk;
                    }
                }
                uint32_t at = __shfl_sync(EG_FULL_MASK, pc, g) + xk - __popc(bits);
                uint32_t off = __shfl_sync(EG_FULL_MASK, pe, g) + xl - len;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (!((bits >> i) & 1u)) continue;
                    queue[at++] = make_uint4(off, r[i] - off, d[i], 0u);
                    off += r[i + 1] - r[i];
                }
            }
        }
        __syncthreads();  // s_cnt, s_edges and s_base are rewritten for the next group
    }
}

// Each warp relaxes an equal share of the round's edges, 128 places per step
// (all columns and weights loaded, then all distances, before any is tested).
// The window holds 32 list entries, one per lane; a place's entry is found
// from the bits of the entries that begin in its 32 places.  A relaxation that
// lowers dist[v] marks v active; the atomicMin's old value is not awaited:
// when another relaxation got below nd first, that one marks v.  Distances are
// read through L1 (popular targets hit there: 1563 -> 1089 us for all rounds
// of RMAT-23); a line read earlier in the kernel can only hold a larger
// distance, which the atomicMin settles.  An edge to the vertex itself never
// lowers its distance.  Bound by the L2 reads of the distances: 161 G
// relaxations a second (63 before, with one edge per lane in flight and each
// list over 256 edges left to a second kernel).
#define EG_SSSP_STEP 4
__global__ void __launch_bounds__(256) k_sssp_push(const uint4 *__restrict__ queue, SsspState *st,
                                                   const uint32_t *__restrict__ col, const uint32_t *__restrict__ wts,
                                                   uint32_t *dist, uint32_t *bm, WRule w) {
    const unsigned long long sel = st->sel;
    const uint32_t cnt = (uint32_t)(sel >> 32), E = (uint32_t)sel;
    const uint32_t lane = threadIdx.x & 31, le = eg_lanemask_lt() | (1u << lane);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->relax += E;
        st->base = st->low == 0xffffffffu ? st->base : st->low;  // distances only grow from round to round's least
        st->low = 0xffffffffu;
    }
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t per = (uint32_t)(((uint64_t)E + warps - 1) / warps);
    per = per < 128u ? 128u : (per + 31u) & ~31u;
    const uint64_t first = (uint64_t)wid * per;
    if (first >= E) return;
    uint32_t p = (uint32_t)first;
    const uint32_t end = E - p > per ? p + per : E;
    uint32_t i0 = eg_list_find(&queue[0].x, 4u, cnt, p);
    for (; p < end; i0 += 32) {
        uint4 q = make_uint4(0xffffffffu, 0u, 0u, 0u);
        if (i0 + lane < cnt) q = __ldg(queue + i0 + lane);
        const uint32_t wend = i0 + 32 < cnt ? __ldg(&queue[i0 + 32].x) : E;
        const uint32_t stop = wend < end ? wend : end;
        for (; p < stop; p = stop - p > 32 * EG_SSSP_STEP ? p + 32 * EG_SSSP_STEP : stop) {  // no wrap at 2^32
            uint32_t v[EG_SSSP_STEP], nd[EG_SSSP_STEP], wt[EG_SSSP_STEP];
#pragma unroll
            for (int k = 0; k < EG_SSSP_STEP; k++) {
                const uint32_t x0 = p + 32 * k;
                const uint32_t starts =
                    __reduce_or_sync(EG_FULL_MASK, q.x - x0 < 32u ? 1u << (q.x - x0) : 0u);
                const uint32_t o = __popc(__ballot_sync(EG_FULL_MASK, q.x < x0)) - 1 + __popc(starts & le);
                const uint32_t at = x0 + lane + __shfl_sync(EG_FULL_MASK, q.y, o);
                const bool on = stop - p > 32u * k + lane;  // x0 + lane may not fit 32 bits
                nd[k] = __shfl_sync(EG_FULL_MASK, q.z, o);
                v[k] = on ? __ldg(col + at) : 0u;
                wt[k] = on ? __ldg(wts + at) : 0u;
            }
            uint32_t cur[EG_SSSP_STEP];
#pragma unroll
            for (int k = 0; k < EG_SSSP_STEP; k++) cur[k] = stop - p > 32u * k + lane ? __ldca(dist + v[k]) : 0u;
#pragma unroll
            for (int k = 0; k < EG_SSSP_STEP; k++) {
                nd[k] = w.add(nd[k], wt[k]);
                if (nd[k] < cur[k]) {
                    atomicMin(dist + v[k], nd[k]);
                    atomicOr(bm + (v[k] >> 5), 1u << (v[k] & 31));
                }
            }
        }
    }
}

__global__ void k_count_reached(const uint32_t *__restrict__ dist, uint64_t len, unsigned long long *out,
                                uint32_t inf) {
    unsigned long long c = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < len; i += (uint64_t)gridDim.x * blockDim.x)
        c += dist[i] != inf;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(EG_FULL_MASK, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

__global__ void k_edge_weights(const uint32_t *__restrict__ rid, const uint32_t *__restrict__ col, uint32_t m,
                               WRule w, uint32_t *__restrict__ out) {
    for (uint64_t p = blockIdx.x * blockDim.x + threadIdx.x; p < m; p += gridDim.x * blockDim.x)
        out[p] = w.weight(__ldg(rid + p), __ldg(col + p));
}

uint32_t blocks_for(eg_ctx *ctx, uint64_t threads) {
    uint64_t b = (threads + 255) / 256;
    uint64_t cap = (uint64_t)ctx->sm_count * 8;
    if (b > cap) b = cap;
    return b ? (uint32_t)b : 1u;
}

int check_weights(const eg_weights *w) {
    if (!w) return EG_OK;
    if (w->rule != EG_W_REF && w->rule != EG_W_HASH && w->rule != EG_W_UNIT && w->rule != EG_W_HASH_F32)
        return eg_fail(EG_EINVAL, "unknown weight rule %d", w->rule);
    if (w->rule == EG_W_HASH && w->hi < w->lo) return eg_fail(EG_EINVAL, "weight range hi < lo");
    return EG_OK;
}

SsspBuckets sssp_buckets(const WRule &w) {
    const uint32_t wmax = w.rule == EG_W_REF ? 18u : w.rule == EG_W_UNIT ? 1u : w.lo + (uint32_t)(w.span - 1);
    const uint32_t wbits = wmax ? 32u - (uint32_t)__builtin_clz(wmax) : 0u;
    return SsspBuckets{w.rule == EG_W_HASH_F32, wbits > EG_SSSP_WBITS ? wbits - EG_SSSP_WBITS : 0u};
}
}  // namespace

int eg_fill_weights(eg_graph *g, const eg_wrule &w, uint32_t *out) {
    eg_ctx *ctx = g->ctx;
    const eg_adj &a = g->csr;
    if (g->m) {
        k_edge_weights<<<blocks_for(ctx, g->m), 256, 0, ctx->stream>>>(bp<uint32_t>(a.rid), bp<uint32_t>(a.col),
                                                                      (uint32_t)g->m, w, out);
        EG_LAUNCHED(ctx);
    }
    return EG_OK;
}

int eg_edge_weights(eg_graph *g, const eg_wrule &w, const uint32_t **out) {
    const uint64_t key[3] = {(uint64_t)w.rule, w.seed, ((uint64_t)w.lo << 32) ^ w.span};
    if (g->wts.p && !memcmp(key, g->wts_key, sizeof(key))) {
        *out = bp<uint32_t>(g->wts);
        return EG_OK;
    }
    EG_TRY(eg_buf_ensure(g->ctx, g->wts, g->m * 4 + 16));
    EG_TRY(eg_fill_weights(g, w, bp<uint32_t>(g->wts)));
    memcpy(g->wts_key, key, sizeof(key));
    *out = bp<uint32_t>(g->wts);
    return EG_OK;
}

// The round loop of eg_sssp as one CUDA graph (a while node over one round).
// Valid while the buffers and the weight array it was captured with (key)
// stay the same.
static int sssp_graph_build(eg_graph *g, const void *const key[8], const uint32_t *wts, const WRule &w, SsspBuckets bk,
                            uint32_t *dist, uint32_t *bm, uint4 *queue, SsspState *st) {
    eg_ctx *ctx = g->ctx;
    eg_bfs_graph &bg = g->s1g;
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
    const uint32_t nw = (g->n + 31) >> 5, blocks = (uint32_t)ctx->sm_count * 8;
    const uint32_t scan = eg_div_up(nw, 256) < blocks ? eg_div_up(nw, 256) : blocks;
    const uint32_t *ptr = bp<uint32_t>(g->csr.ptr), *col = bp<uint32_t>(g->csr.col);
    EG_CUDA(cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    const uint32_t hmost = (uint32_t)ctx->sm_count * EG_SSSP_HB;
    k_sssp_hist<<<scan < hmost ? scan : hmost, 256, 0, ctx->stream>>>(bm, nw, ptr, dist, bk, st, handle);
    k_sssp_select<<<scan, 256, 0, ctx->stream>>>(bm, nw, ptr, dist, bk, st, queue);
    k_sssp_push<<<blocks, 256, 0, ctx->stream>>>(queue, st, col, wts, dist, bm, w);
    cudaError_t ce = cudaStreamEndCapture(ctx->stream, &body);
    if (ce != cudaSuccess) return eg_fail(EG_ECUDA, "SSSP capture: %s", cudaGetErrorString(ce));
    cudaGraphExec_t exec = nullptr;
    EG_TRY(eg_graph_instantiate(ctx, &exec, graph));
    bg.exec = exec;
    for (int i = 0; i < 8; i++) bg.key[i] = key[i];
    return EG_OK;
}

extern "C" int eg_sssp(eg_graph *g, uint32_t root, const eg_weights *wrule_in, uint32_t *dist_out,
                       eg_sssp_stats *stats) {
    if (!g) return eg_fail(EG_EINVAL, "NULL graph");
    if (root >= g->n) return eg_fail(EG_EINVAL, "root %u >= n %u", root, g->n);
    if (!(g->built & EG_LAYOUT_CSR)) return eg_fail(EG_ENOTBUILT, "SSSP needs the CSR");
    EG_TRY(check_weights(wrule_in));
    eg_ctx *ctx = g->ctx;
    EG_CUDA(cudaSetDevice(ctx->device));
    const uint32_t n = g->n, nw = (n + 31) >> 5;
    const WRule w = eg_make_wrule(wrule_in);
    const uint32_t *wts = nullptr;
    EG_TRY(eg_edge_weights(g, w, &wts));
    EG_TRY(eg_buf_ensure(ctx, g->dist, (uint64_t)n * 4));
    // work: list [n uint4] | active bits | state | reached
    const uint64_t off_bm = 4ull * n, off_st = (off_bm + nw + 7) & ~7ull, off_cnt = off_st + sizeof(SsspState) / 4;
    EG_TRY(eg_buf_ensure(ctx, g->sssp_work, (off_cnt + 4) * 4));
    uint32_t *wk = bp<uint32_t>(g->sssp_work);
    uint4 *queue = reinterpret_cast<uint4 *>(wk);
    uint32_t *bm = wk + off_bm;
    SsspState *st = reinterpret_cast<SsspState *>(wk + off_st);
    unsigned long long *dcount = reinterpret_cast<unsigned long long *>(wk + off_cnt);
    uint32_t *dist = bp<uint32_t>(g->dist);
    const SsspBuckets bk = sssp_buckets(w);
    const void *key[8] = {wk, wts, dist, g->csr.ptr.p, g->csr.col.p, (const void *)(uintptr_t)w.rule,
                          (const void *)(uintptr_t)bk.shift, (const void *)(uintptr_t)n};
    eg_bfs_graph &bg = g->s1g;
    bool same = bg.exec != nullptr;
    for (int i = 0; i < 8 && same; i++) same = bg.key[i] == key[i];
    if (!same) EG_TRY(sssp_graph_build(g, key, wts, w, bk, dist, bm, queue, st));
    EG_CUDA(cudaEventRecord(ctx->ev0, ctx->stream));
    const uint32_t ib = blocks_for(ctx, n > 4 * EG_SSSP_BUCKETS ? n : 4 * EG_SSSP_BUCKETS);
    k_sssp_init<<<ib, 256, 0, ctx->stream>>>(n, nw, dist, root, bm, st, w.inf(), n + 16u);
    EG_LAUNCHED(ctx);
    EG_CUDA(cudaGraphLaunch(bg.exec, ctx->stream));
    ctx->launches += 1;
    EG_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
    if (dist_out) EG_CUDA(cudaMemcpyAsync(dist_out, dist, (uint64_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    unsigned long long *h = (unsigned long long *)ctx->h_pinned;
    SsspState *hs = reinterpret_cast<SsspState *>(h + 2);
    if (stats) {
        EG_TRY(eg_zero(ctx, dcount, 8, ctx->stream));
        k_count_reached<<<blocks_for(ctx, n), 256, 0, ctx->stream>>>(dist, n, dcount, w.inf());
        EG_LAUNCHED(ctx);
        EG_TRY(eg_readback(ctx, h, dcount, 8, ctx->stream));
    }
    EG_TRY(eg_readback_wait(ctx, hs, st, offsetof(SsspState, hist), ctx->stream));
    if (dist_out || stats) EG_CUDA(cudaStreamSynchronize(ctx->stream));
    if (hs->err) return eg_fail(EG_ETIMEOUT, "SSSP did not converge");
    if (stats) {
        stats->reached = (uint32_t)h[0];
        stats->rounds = (int)hs->rounds;
        stats->relaxations = hs->relax;
        EG_CUDA(cudaEventElapsedTime(&stats->ms, ctx->ev0, ctx->ev1));
    }
    return EG_OK;
}

// ============================================================== multi-source
// dist is vertex-major: dist[v * kp + s], kp = k rounded up to 4.  An item is a
// vertex and a word of 32 sources; act[v * kw + j] holds the sources of word j
// whose distance at v dropped since the item's list was last relaxed.
//
// The rounds are ordered like the single source's, by item: an item's key is
// the least of its active sources' distances, each taken from that source's
// own base (a lower bound of its active distances).  Distances from different
// sources differ mostly by an offset, so the sources of a word reach a vertex
// at about the same key and share the visit: on RMAT-15, 32 sources, weights
// 1..255, the lists are read 3.5 times per edge and word and each (edge,
// source) pair is relaxed 1.8 times, against 7.9 and 3.7 when every active item
// goes in every round, and 7 and 1.1 when each source goes by its own
// threshold (a CPU count of the rounds).  After n + 16 ordered rounds every
// active item goes in every round: n more at most.
namespace {
// Places (edges of items) of a round at least.  Directed RMAT, 1,000,003
// vertices, 64 sources: 2^19 43 rounds 9.3 ms, 2^20 26 rounds 7.5, 2^21 22
// rounds 7.1, with the distances' copy to the host (1.3 ms).
#define EG_MSSSP_MIN_WORK (1u << 21)
struct MsState {
    unsigned long long sel;    // this round's list: items << 32 | places
    unsigned long long relax;  // (edge, active source) pairs listed so far
    uint32_t last;             // last bucket of the round
    uint32_t done;             // CTAs of the histogram that are finished
    uint32_t rounds, limit, err;
    uint32_t ordered;          // rounds up to this one are ordered
    uint32_t pad[2];
    uint32_t hist[EG_SSSP_BUCKETS];
};

__global__ void k_msssp_init(uint64_t rows4, uint64_t items, uint4 *dist, uint32_t *act, uint32_t kp, uint32_t *base,
                             uint32_t *low, MsState *st, uint32_t inf, uint32_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, i0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    for (uint64_t i = i0; i < rows4; i += stride) dist[i] = make_uint4(inf, inf, inf, inf);
    for (uint64_t i = i0; i < items; i += stride) act[i] = 0;
    for (uint64_t i = i0; i < kp; i += stride) base[i] = low[i] = 0;  // the roots' distances
    for (uint64_t i = i0; i < EG_SSSP_BUCKETS; i += stride) st->hist[i] = 0;
    if (i0 == 0) {
        st->sel = st->relax = 0;
        st->last = EG_SSSP_BUCKETS - 1;
        st->done = 0;
        st->rounds = 0;
        st->ordered = n + 16u;
        st->limit = n > 0x7fffffe0u ? 0xffffffffu : 2u * n + 32u;
        st->err = 0;
    }
}

__global__ void k_msssp_roots(const uint32_t *roots, int k, uint32_t kp, uint32_t kw, uint32_t *dist, uint32_t *act) {
    for (int s = threadIdx.x; s < k; s += blockDim.x) {
        const uint32_t r = roots[s];
        dist[(uint64_t)r * kp + s] = 0;
        atomicOr(act + (uint64_t)r * kw + (s >> 5), 1u << (s & 31));
    }
}

// Words of the active items in flight per lane: most are zero where entries are
// few (4 sources, n = 16.8 M, 4 K entries: a call 330 us one by one, 314, 305 and
// 310 with 2, 4 and 8; 64 sources 2624 -> 2530).  With 8 the dense passes lose:
// 1,000,003 vertices, 64 sources 6.16 -> 6.39 ms, with 4 6.14.
#define EG_MSSSP_HWORDS 4
// Places per bucket of the active items' keys, and the keys themselves (a
// group of 8 lanes per item, four sources per lane).  Source s's base is the
// least of the distances relaxations lowered last round (low[s]) and, where
// items were left out then, the end of that round's buckets.  The last CTA
// picks this round's last bucket and sets the loop condition.
__global__ void __launch_bounds__(256) k_msssp_hist(const uint32_t *__restrict__ act, uint64_t items, uint32_t kw,
                                                    uint32_t kp, const uint32_t *__restrict__ ptr,
                                                    const uint32_t *__restrict__ dist, SsspBuckets bk, MsState *st,
                                                    uint32_t *base, uint32_t *low, uint16_t *__restrict__ keys,
                                                    uint32_t inf, cudaGraphConditionalHandle handle) {
    __shared__ uint32_t s_hist[EG_SSSP_BUCKETS];
    __shared__ __align__(16) uint32_t s_base[1024];
    __shared__ uint32_t s_last;
    __shared__ unsigned long long s_sum[8];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane >> 3, sl = lane & 7;
    for (uint32_t i = threadIdx.x; i < EG_SSSP_BUCKETS; i += 256) s_hist[i] = 0;
    const uint32_t prev = st->last;
    for (uint32_t i = threadIdx.x; i < kp; i += 256)
        s_base[i] = prev == EG_SSSP_BUCKETS - 1 ? low[i] : min(low[i], bk.end(base[i], prev, inf));
    __syncthreads();
    const uint64_t stride = gridDim.x * 256ull;
    for (uint64_t it0 = (blockIdx.x * 8ull + warp) * 32; it0 < items; it0 += EG_MSSSP_HWORDS * stride) {
        uint32_t words[EG_MSSSP_HWORDS];
#pragma unroll
        for (int j = 0; j < EG_MSSSP_HWORDS; j++)
            words[j] = it0 + j * stride + lane < items ? __ldg(act + it0 + j * stride + lane) : 0u;
#pragma unroll
        for (int j = 0; j < EG_MSSSP_HWORDS; j++) {
            const uint32_t word = words[j];
            const uint32_t some = __ballot_sync(EG_FULL_MASK, word != 0u);
            if (!some) continue;
#pragma unroll 1
            for (uint32_t i = 0; i < 8; i++) {
                if (!((some >> (4 * i)) & 15u)) continue;
                const uint32_t a = __shfl_sync(EG_FULL_MASK, word, 4 * i + grp);
                const uint32_t item = (uint32_t)(it0 + j * stride) + 4 * i + grp;
                const uint32_t v = item / kw, s0 = 32 * (item - v * kw) + 4 * sl;
                const uint32_t nib = (a >> (4 * sl)) & 15u;
                uint32_t key = EG_SSSP_BUCKETS - 1;
                if (nib) {
                    const uint4 d = __ldg(reinterpret_cast<const uint4 *>(dist + (uint64_t)v * kp + s0));
                    const uint4 b = *reinterpret_cast<const uint4 *>(s_base + s0);
                    if (nib & 1u) key = min(key, bk.of(max(d.x, b.x), b.x));
                    if (nib & 2u) key = min(key, bk.of(max(d.y, b.y), b.y));
                    if (nib & 4u) key = min(key, bk.of(max(d.z, b.z), b.z));
                    if (nib & 8u) key = min(key, bk.of(max(d.w, b.w), b.w));
                }
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) key = min(key, __shfl_xor_sync(EG_FULL_MASK, key, o));
                if (a && sl == 0) {
                    keys[item] = (uint16_t)key;
                    const uint32_t len = __ldg(ptr + v + 1) - __ldg(ptr + v);
                    if (len) atomicAdd(&s_hist[key], len);
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < EG_SSSP_BUCKETS; i += 256)
        if (s_hist[i]) atomicAdd(&st->hist[i], s_hist[i]);
    __threadfence();
    __syncthreads();  // every thread's adds are out before the CTA counts as done
    if (threadIdx.x == 0) s_last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // the last CTA: the bases for the next round, four buckets per thread
    for (uint32_t i = threadIdx.x; i < kp; i += 256) {
        base[i] = s_base[i];
        low[i] = inf;
    }
    unsigned long long c[4], sum = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        c[i] = sum += __ldcg(&st->hist[threadIdx.x * 4 + i]);
        st->hist[threadIdx.x * 4 + i] = 0;
    }
    uint32_t last;
    const unsigned long long total = sssp_pick(c, sum, EG_MSSSP_MIN_WORK, s_sum, &s_last, &last);
    if (threadIdx.x == 0) {
        st->done = 0;
        st->sel = 0;
        if (total) st->rounds += 1;
        st->last = st->rounds > st->ordered ? EG_SSSP_BUCKETS - 1 : last;
        const bool over = total && st->rounds > st->limit;
        if (over) st->err = 1;
        cudaGraphSetConditional(handle, total && !over ? 1u : 0u);
    }
}

// Lists the round's items (x = first place among the round's places, y = the
// item) and clears their words; four items per thread.
__global__ void __launch_bounds__(256) k_msssp_select(uint32_t *__restrict__ act, const uint16_t *__restrict__ keys,
                                                      uint64_t items, uint32_t kw, const uint32_t *__restrict__ ptr,
                                                      MsState *st, uint2 *__restrict__ queue) {
    __shared__ uint32_t s_cnt[8], s_edges[8];
    __shared__ unsigned long long s_base, s_relax;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t last = st->last;
    if (threadIdx.x == 0) s_relax = 0;
    unsigned long long relax = 0;
    // uniform trip count per CTA; the arrays' ends are padded to 16 bytes
    for (uint64_t c0 = blockIdx.x * 1024ull; c0 < items; c0 += gridDim.x * 1024ull) {
        const uint64_t i0 = c0 + threadIdx.x * 4;
        uint32_t a[4] = {0u, 0u, 0u, 0u}, len[4] = {0u, 0u, 0u, 0u};
        if (i0 < items) {
            const uint4 q = *reinterpret_cast<const uint4 *>(act + i0);
            a[0] = q.x;
            a[1] = i0 + 1 < items ? q.y : 0u;
            a[2] = i0 + 2 < items ? q.z : 0u;
            a[3] = i0 + 3 < items ? q.w : 0u;
        }
        if (!__syncthreads_or((a[0] | a[1] | a[2] | a[3]) != 0u)) continue;
        uint32_t cnt = 0, edges = 0;
        if (a[0] | a[1] | a[2] | a[3]) {
            const ushort4 key = __ldg(reinterpret_cast<const ushort4 *>(keys + i0));
            const uint32_t kk[4] = {key.x, key.y, key.z, key.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (!a[i]) continue;
                const uint32_t v = ((uint32_t)i0 + i) / kw;
                len[i] = __ldg(ptr + v + 1) - __ldg(ptr + v);
                if (len[i] && kk[i] > last) {  // left for a later round
                    len[i] = 0;
                    continue;
                }
                act[i0 + i] = 0;
                cnt += len[i] != 0;
                edges += len[i];
                relax += (unsigned long long)len[i] * __popc(a[i]);
            }
        }
        uint32_t xc = cnt, xe = edges;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t yc = __shfl_up_sync(EG_FULL_MASK, xc, o), ye = __shfl_up_sync(EG_FULL_MASK, xe, o);
            if (lane >= (uint32_t)o) {
                xc += yc;
                xe += ye;
            }
        }
        if (lane == 31) {
            s_cnt[warp] = xc;
            s_edges[warp] = xe;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t tc = 0, te = 0;
            for (int i = 0; i < 8; i++) {
                const uint32_t p = s_cnt[i], q = s_edges[i];
                s_cnt[i] = tc;
                s_edges[i] = te;
                tc += p;
                te += q;
            }
            // one word for both sums (m * kw < 2^32), so that they keep the same order
            s_base = tc ? atomicAdd(&st->sel, ((unsigned long long)tc << 32) | te) : 0ull;
        }
        __syncthreads();
        uint32_t at = (uint32_t)(s_base >> 32) + s_cnt[warp] + xc - cnt;
        uint32_t off = (uint32_t)s_base + s_edges[warp] + xe - edges;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (!len[i]) continue;
            queue[at++] = make_uint2(off, (uint32_t)i0 + i);
            off += len[i];
        }
        __syncthreads();  // s_cnt, s_edges and s_base are rewritten for the next 1024
    }
    __syncthreads();
    if (relax) atomicAdd(&s_relax, relax);
    __syncthreads();
    if (threadIdx.x == 0 && s_relax) atomicAdd(&st->relax, s_relax);
}

// Each warp takes an equal share of the round's places (edges of listed
// items), 32 at a time: a lane finds its place's item and loads its column
// and weight, then groups of 8 lanes relax one place each, four sources per
// lane, EG_MSSSP_ROWS places per group in flight.  All sources of the word
// are relaxed, active or not (a distance read at the item is that of a path
// either way), and the item's row is read again for every place, mostly from
// L1, so that no place waits for another.  Bound by the L2 reads and
// atomics of the rows: 30 G places a second (10 G before, when a warp walked
// one item after another and hubs went through a second kernel); one place
// per group in flight 4.42 ms, two 4.06, four (more registers) 5.81 for all
// rounds of 1,000,003 vertices, 64 sources.
#define EG_MSSSP_ROWS 2
__global__ void __launch_bounds__(256) k_msssp_push(const uint2 *__restrict__ queue, const MsState *st,
                                                    const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ col,
                                                    const uint32_t *__restrict__ wts, uint32_t kw, uint32_t kp,
                                                    uint32_t *dist, uint32_t *act, uint32_t *low, WRule w) {
    __shared__ __align__(16) uint32_t s_low[1024];
    const unsigned long long sel = st->sel;
    const uint32_t cnt = (uint32_t)(sel >> 32), E = (uint32_t)sel;
    const uint32_t lane = threadIdx.x & 31, le = eg_lanemask_lt() | (1u << lane), grp = lane >> 3, sl = lane & 7;
    const uint32_t inf = w.inf();
    for (uint32_t i = threadIdx.x; i < kp; i += 256) s_low[i] = inf;
    __syncthreads();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t per = (uint32_t)(((uint64_t)E + warps - 1) / warps);
    per = (per + 31u) & ~31u;
    const uint64_t first = (uint64_t)wid * per;
    uint32_t p = first < E ? (uint32_t)first : E;
    const uint32_t end = E - p > per ? p + per : E;
    uint32_t i0 = p < end ? eg_list_find(&queue[0].x, 2u, cnt, p) : 0u;
    for (; p < end; i0 += 32) {
        uint32_t q_off = 0xffffffffu, q_u = 0, q_j = 0, q_add = 0;
        if (i0 + lane < cnt) {
            const uint2 q = __ldg(queue + i0 + lane);
            q_off = q.x;
            q_u = q.y / kw;
            q_j = q.y - q_u * kw;
            q_add = __ldg(ptr + q_u) - q_off;
        }
        const uint32_t wend = i0 + 32 < cnt ? __ldg(&queue[i0 + 32].x) : E;
        const uint32_t stop = wend < end ? wend : end;
        for (; p < stop; p = stop - p > 32u ? p + 32u : stop) {
            const uint32_t starts = __reduce_or_sync(EG_FULL_MASK, q_off - p < 32u ? 1u << (q_off - p) : 0u);
            const uint32_t o = __popc(__ballot_sync(EG_FULL_MASK, q_off < p)) - 1 + __popc(starts & le);
            const uint32_t at = p + lane + __shfl_sync(EG_FULL_MASK, q_add, o);
            const uint32_t u = __shfl_sync(EG_FULL_MASK, q_u, o), j = __shfl_sync(EG_FULL_MASK, q_j, o);
            const bool on = p + lane < stop;
            const uint32_t v = on ? __ldg(col + at) : 0u, wt = on ? __ldg(wts + at) : 0u;
            const uint32_t left = stop - p < 32u ? stop - p : 32u;
            for (uint32_t i = 0; i < left; i += 4 * EG_MSSSP_ROWS) {
                uint4 du[EG_MSSSP_ROWS], dv[EG_MSSSP_ROWS];
                uint32_t *row[EG_MSSSP_ROWS];
                uint32_t vv[EG_MSSSP_ROWS], jj[EG_MSSSP_ROWS], ww[EG_MSSSP_ROWS];
                bool ok[EG_MSSSP_ROWS];
#pragma unroll
                for (int r = 0; r < EG_MSSSP_ROWS; r++) {
                    const uint32_t src = (i + 4 * r + grp) & 31u;
                    const uint32_t uu = __shfl_sync(EG_FULL_MASK, u, src);
                    jj[r] = __shfl_sync(EG_FULL_MASK, j, src);
                    vv[r] = __shfl_sync(EG_FULL_MASK, v, src);
                    ww[r] = __shfl_sync(EG_FULL_MASK, wt, src);
                    const uint32_t s0 = 32 * jj[r] + 4 * sl;
                    ok[r] = i + 4 * r + grp < left && s0 < kp;
                    row[r] = dist + (uint64_t)vv[r] * kp + s0;
                    if (ok[r]) {
                        du[r] = __ldca(reinterpret_cast<const uint4 *>(dist + (uint64_t)uu * kp + s0));
                        dv[r] = __ldca(reinterpret_cast<const uint4 *>(row[r]));
                    }
                }
#pragma unroll
                for (int r = 0; r < EG_MSSSP_ROWS; r++) {
                    uint32_t nib = 0;
                    if (ok[r]) {
                        const uint32_t s0 = 32 * jj[r] + 4 * sl;
                        const uint32_t nd[4] = {w.add(du[r].x, ww[r]), w.add(du[r].y, ww[r]), w.add(du[r].z, ww[r]),
                                                w.add(du[r].w, ww[r])};
                        const uint32_t cur[4] = {dv[r].x, dv[r].y, dv[r].z, dv[r].w};
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            if (nd[c] < cur[c]) {
                                atomicMin(row[r] + c, nd[c]);
                                nib |= 1u << c;
                                if (nd[c] < s_low[s0 + c]) atomicMin(&s_low[s0 + c], nd[c]);
                            }
                        }
                    }
                    uint32_t mask = nib << (4 * sl);
                    if (!__any_sync(EG_FULL_MASK, mask != 0u)) continue;
#pragma unroll
                    for (int o2 = 1; o2 < 8; o2 <<= 1) mask |= __shfl_xor_sync(EG_FULL_MASK, mask, o2);
                    if (sl == 0 && mask) atomicOr(act + (uint64_t)vv[r] * kw + jj[r], mask);
                }
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kp; i += 256)
        if (s_low[i] < __ldcg(low + i)) atomicMin(low + i, s_low[i]);
}

// out[s][v] = dvk[v * kp + s] for s < k.
__global__ void k_transpose_dist(const uint32_t *__restrict__ dvk, uint32_t n, int k, uint32_t kp,
                                 uint32_t *__restrict__ dkv) {
    __shared__ uint32_t t[32][33];
    uint32_t v0 = blockIdx.x * 32, s0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        uint32_t v = v0 + r, s = s0 + threadIdx.x;
        t[r][threadIdx.x] = (v < n && s < (uint32_t)k) ? dvk[(uint64_t)v * kp + s] : 0u;
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += blockDim.y) {
        uint32_t s = s0 + r, v = v0 + threadIdx.x;
        if (v < n && s < (uint32_t)k) dkv[(uint64_t)s * n + v] = t[threadIdx.x][r];
    }
}
}  // namespace

// The round loop of eg_sssp_multi as one CUDA graph (a while node over one
// round).  Valid while the buffers, the batch size and the weight array it
// was captured with (key) stay the same.
static int msssp_graph_build(eg_graph *g, const void *const key[8], const uint32_t *wts, uint32_t kp, uint32_t kw,
                             const WRule &w, SsspBuckets bk, uint32_t *dist, uint32_t *act, uint16_t *keys, uint2 *queue,
                             uint32_t *base, uint32_t *low, MsState *st) {
    eg_ctx *ctx = g->ctx;
    eg_bfs_graph &bg = g->ssg;
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
    const uint64_t items = (uint64_t)g->n * kw;
    const uint32_t blocks = (uint32_t)ctx->sm_count * 8;
    const uint32_t hb = eg_div_up(items, 256) < blocks ? eg_div_up(items, 256) : blocks;
    const uint32_t sb = eg_div_up(items, 1024) < blocks ? eg_div_up(items, 1024) : blocks;
    const uint32_t *ptr = bp<uint32_t>(g->csr.ptr), *col = bp<uint32_t>(g->csr.col);
    EG_CUDA(cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
    k_msssp_hist<<<hb, 256, 0, ctx->stream>>>(act, items, kw, kp, ptr, dist, bk, st, base, low, keys, w.inf(), handle);
    k_msssp_select<<<sb, 256, 0, ctx->stream>>>(act, keys, items, kw, ptr, st, queue);
    k_msssp_push<<<blocks, 256, 0, ctx->stream>>>(queue, st, ptr, col, wts, kw, kp, dist, act, low, w);
    cudaError_t ce = cudaStreamEndCapture(ctx->stream, &body);
    if (ce != cudaSuccess) return eg_fail(EG_ECUDA, "batched SSSP capture: %s", cudaGetErrorString(ce));
    cudaGraphExec_t exec = nullptr;
    EG_TRY(eg_graph_instantiate(ctx, &exec, graph));
    bg.exec = exec;
    for (int i = 0; i < 8; i++) bg.key[i] = key[i];
    return EG_OK;
}

extern "C" int eg_sssp_multi(eg_graph *g, const uint32_t *roots, int k, const eg_weights *wrule_in,
                             uint32_t *dist_out, eg_sssp_stats *stats) {
    if (!g || !roots) return eg_fail(EG_EINVAL, "NULL argument");
    if (k < 1 || k > 1024) return eg_fail(EG_EINVAL, "k=%d: batched SSSP takes 1..1024 sources", k);
    if (!(g->built & EG_LAYOUT_CSR)) return eg_fail(EG_ENOTBUILT, "SSSP needs the CSR");
    EG_TRY(check_weights(wrule_in));
    for (int s = 0; s < k; s++)
        if (roots[s] >= g->n) return eg_fail(EG_EINVAL, "root %u >= n", roots[s]);
    if (k == 1) return eg_sssp(g, roots[0], wrule_in, dist_out, stats);
    eg_ctx *ctx = g->ctx;
    EG_CUDA(cudaSetDevice(ctx->device));
    const uint32_t n = g->n;
    const WRule w = eg_make_wrule(wrule_in);
    const uint32_t *wts = nullptr;
    EG_TRY(eg_edge_weights(g, w, &wts));
    if ((uint64_t)n * ((k + 31) / 32) >= 0xffffffffull) return eg_fail(EG_EINVAL, "n * ceil(k/32) must be < 2^32");
    // a round's places are counted in 32 bits: at most that many words at once
    const uint64_t most = g->m ? 0xffffff00ull / g->m : 32;
    const int kb_max = most >= 32 ? 1024 : (int)(32 * (most ? most : 1));
    const SsspBuckets bk = sssp_buckets(w);
    float ms = 0.f;
    uint64_t reached = 0, relax = 0;
    int rounds = 0;
    if (dist_out) EG_TRY(eg_buf_ensure(ctx, g->dist, (uint64_t)n * k * 4));
    for (int k0 = 0; k0 < k; k0 += kb_max) {
        const int kb = k - k0 < kb_max ? k - k0 : kb_max;
        const uint32_t kw = (uint32_t)((kb + 31) / 32), kp = ((uint32_t)kb + 3u) & ~3u;
        const uint64_t items = (uint64_t)n * kw;
        // work: dist[n * kp] | act[items] | keys[items u16] | list[items uint2] | base, low [kp] | roots | state | reached
        auto up = [](uint64_t x) { return (x + 7) & ~7ull; };
        const uint64_t off_act = up((uint64_t)n * kp), off_keys = up(off_act + items), off_q = up(off_keys + (items + 1) / 2),
                       off_base = up(off_q + 2 * items), off_low = off_base + up(kp), off_roots = off_low + up(kp),
                       off_st = off_roots + 1024, off_cnt = off_st + up(sizeof(MsState) / 4);
        EG_TRY(eg_buf_ensure(ctx, g->sssp_work, (off_cnt + 4) * 4));
        uint32_t *wk = bp<uint32_t>(g->sssp_work);
        uint32_t *dist = wk, *act = wk + off_act, *base = wk + off_base, *low = wk + off_low, *d_roots = wk + off_roots;
        uint16_t *keys = reinterpret_cast<uint16_t *>(wk + off_keys);
        uint2 *queue = reinterpret_cast<uint2 *>(wk + off_q);
        MsState *st = reinterpret_cast<MsState *>(wk + off_st);
        unsigned long long *dcount = reinterpret_cast<unsigned long long *>(wk + off_cnt);
        const void *key[8] = {wk, wts, g->csr.col.p, g->csr.ptr.p, (const void *)(uintptr_t)kb,
                              (const void *)(uintptr_t)w.rule, (const void *)(uintptr_t)bk.shift,
                              (const void *)(uintptr_t)n};
        eg_bfs_graph &bg = g->ssg;
        bool same = bg.exec != nullptr;
        for (int i = 0; i < 8 && same; i++) same = bg.key[i] == key[i];
        if (!same) EG_TRY(msssp_graph_build(g, key, wts, kp, kw, w, bk, dist, act, keys, queue, base, low, st));
        EG_CUDA(cudaMemcpyAsync(d_roots, roots + k0, (uint64_t)kb * 4, cudaMemcpyHostToDevice, ctx->stream));
        EG_CUDA(cudaEventRecord(ctx->ev0, ctx->stream));
        k_msssp_init<<<blocks_for(ctx, (uint64_t)n * kp / 4 + EG_SSSP_BUCKETS), 256, 0, ctx->stream>>>(
            (uint64_t)n * kp / 4, items, reinterpret_cast<uint4 *>(dist), act, kp, base, low, st, w.inf(), n);
        EG_LAUNCHED(ctx);
        k_msssp_roots<<<1, 256, 0, ctx->stream>>>(d_roots, kb, kp, kw, dist, act);
        EG_LAUNCHED(ctx);
        EG_CUDA(cudaGraphLaunch(bg.exec, ctx->stream));
        ctx->launches += 1;
        EG_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
        if (dist_out) {
            dim3 grid(eg_div_up(n, 32), eg_div_up((uint64_t)kb, 32)), block(32, 8);
            k_transpose_dist<<<grid, block, 0, ctx->stream>>>(dist, n, kb, kp, bp<uint32_t>(g->dist) + (uint64_t)k0 * n);
            EG_LAUNCHED(ctx);
            EG_CUDA(cudaMemcpyAsync(dist_out + (uint64_t)k0 * n, bp<uint32_t>(g->dist) + (uint64_t)k0 * n,
                                    (uint64_t)n * kb * 4, cudaMemcpyDeviceToHost, ctx->stream));
        }
        unsigned long long *h = (unsigned long long *)ctx->h_pinned;
        MsState *hs = reinterpret_cast<MsState *>(h + 2);
        if (stats) {
            EG_TRY(eg_zero(ctx, dcount, 8, ctx->stream));
            k_count_reached<<<blocks_for(ctx, (uint64_t)n * kp), 256, 0, ctx->stream>>>(dist, (uint64_t)n * kp, dcount,
                                                                                       w.inf());
            EG_LAUNCHED(ctx);
            EG_TRY(eg_readback(ctx, h, dcount, 8, ctx->stream));
        }
        EG_TRY(eg_readback(ctx, hs, st, offsetof(MsState, hist), ctx->stream));
        EG_CUDA(cudaStreamSynchronize(ctx->stream));
        if (hs->err) return eg_fail(EG_ETIMEOUT, "batched SSSP did not converge");
        if (stats) {
            float t = 0.f;
            EG_CUDA(cudaEventElapsedTime(&t, ctx->ev0, ctx->ev1));
            ms += t;
            reached += h[0];
            relax += hs->relax;
            rounds = (int)hs->rounds > rounds ? (int)hs->rounds : rounds;
        }
    }
    if (stats) {
        stats->reached = (uint32_t)(reached > 0xffffffffull ? 0xffffffffull : reached);
        stats->rounds = rounds;
        stats->relaxations = relax;
        stats->ms = ms;
    }
    return EG_OK;
}
