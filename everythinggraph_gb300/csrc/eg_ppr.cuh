// Kernels of the batched personalised PageRank (see eg_ppr.cu), shared with
// the query server.  Internal linkage: each translation unit has its copy.
#pragma once
#include "eg_internal.cuh"

#define EG_PPR_LANES 32
// entries per item: a whole row has at most EG_PPR_PART - 1 (its length order
// is then one 9-bit sort pass), longer rows are cut into parts of EG_PPR_PART
#define EG_PPR_PART 512u
// resident CTAs per SM of k_ppr_rows (48 registers).  RMAT-20 undirected, 32
// queries: 3 325 us a sweep, 4 275, 5 249
#define EG_PPR_MINB 5

namespace {

struct PprQ {  // per-query state (device)
    double residual;
    double dangling;
    float tol;
    int iters;
    int max_iters;
    int done;
    int nseeds;
    int active;  // lane in use
};

__device__ __forceinline__ float4 eg_f4add(float4 a, float4 b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
// Eight rows' sum.  Long sums take them eight by eight: a chain of an addition
// per eight entries rounds less (511 equal entries one by one: off by 7.6e-6 of
// the sum, this way by 5e-8).
__device__ __forceinline__ float4 eg_f4sum8(const float4 (&x)[8]) {
    float4 s = x[0];
#pragma unroll
    for (int i = 1; i < 8; i++) s = eg_f4add(s, x[i]);
    return s;
}
__device__ __forceinline__ float4 eg_f4shfl(unsigned mask, float4 v, int src) {
    return make_float4(__shfl_sync(mask, v.x, src), __shfl_sync(mask, v.y, src), __shfl_sync(mask, v.z, src),
                       __shfl_sync(mask, v.w, src));
}

// Y[v][q] = sum over CSC entries of row v of X[u][q], over the work list of
// eg_ppr_plan: items of at most EG_PPR_PART entries, longest first.  Items
// [0, nlong) are the parts of the rows with more entries than that, their sums
// go to part rows that k_ppr_fixup adds up; the others are whole rows.
//
// The warp is four groups of 8 lanes; lane s of a group holds queries
// 4s..4s+3 (one 16-byte load brings a group a whole 128-byte row of X), and a
// group takes one item, 8 entries per step with their 8 row loads in flight.
// An item is summed in entry order, eight entries at a time, so a query's bits
// depend on the graph alone.  Items of a warp have nearly equal lengths and no entry needs a row
// id or a test for the row's end; the next item's place is loaded while the
// current one is summed.  Bound by the latency of the L2 row reads (a
// sweep of undirected RMAT-20: 249 us, 15 TB/s of rows; 413 when each warp
// walked a range of entries, testing every entry's row id: 9.6 warp
// instructions per entry).
__global__ void __launch_bounds__(256, EG_PPR_MINB) k_ppr_rows(const uint32_t *__restrict__ ptr,
                                                               const uint32_t *__restrict__ col,
                                                               const uint4 *__restrict__ longs, uint32_t nlong,
                                                               const uint32_t *__restrict__ order, uint32_t nrows,
                                                               const float *__restrict__ X, float *__restrict__ Y,
                                                               float *__restrict__ part) {
    const uint32_t lane = threadIdx.x & 31, grp = lane >> 3, sl = lane & 7;
    const float4 *__restrict__ X4 = reinterpret_cast<const float4 *>(X) + sl;
    const uint32_t items = nlong + nrows, step = ((gridDim.x * blockDim.x) >> 5) * 4;
    struct Item {
        uint32_t begin, len, dst;
    };
    auto row_at = [&](uint32_t i) { return i >= nlong && i < items ? __ldg(order + (i - nlong)) : 0u; };
    auto item_at = [&](uint32_t i, uint32_t row) {  // row: row_at(i)
        Item t = {0u, 0u, row};
        if (i < nlong) {
            const uint4 l = __ldg(longs + i);
            t = {l.x, l.y, l.z};
        } else if (i < items) {
            t.begin = __ldg(ptr + row);
            t.len = __ldg(ptr + row + 1) - t.begin;
        }
        return t;
    };
    // the warp's four items, i0 .. i0 + 3 (lengths 0 past the end), together
    uint32_t i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 4;
    Item cur = item_at(i0 + grp, row_at(i0 + grp));
    uint32_t row1 = row_at(i0 + step + grp);
    for (; i0 < items; i0 += step) {
        uint32_t my_c = sl < cur.len ? __ldg(col + cur.begin + sl) : 0u;
        const Item nxt = item_at(i0 + step + grp, row1);
        row1 = row_at(i0 + 2 * step + grp);
        const uint32_t most = __reduce_max_sync(EG_FULL_MASK, cur.len), least = __reduce_min_sync(EG_FULL_MASK, cur.len);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (uint32_t b = 0; b < most; b += 8) {
            const uint32_t e = b + 8 + sl;
            const uint32_t next_c = e < cur.len ? __ldg(col + cur.begin + e) : 0u;
            float4 xv[8];
            if (b + 8 <= least) {
#pragma unroll
                for (int q = 0; q < 8; q++)
                    xv[q] = __ldg(X4 + (uint64_t)__shfl_sync(EG_FULL_MASK, my_c, q, 8) * (EG_PPR_LANES / 4));
                acc = eg_f4add(acc, eg_f4sum8(xv));
            } else {
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const uint32_t u = __shfl_sync(EG_FULL_MASK, my_c, q, 8);
                    xv[q] = b + q < cur.len ? __ldg(X4 + (uint64_t)u * (EG_PPR_LANES / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                float4 s = xv[0];
#pragma unroll
                for (int q = 1; q < 8; q++)
                    if (b + q < cur.len) s = eg_f4add(s, xv[q]);
                acc = eg_f4add(acc, s);
            }
            my_c = next_c;
        }
        if (i0 + grp < items) {
            float4 *out = reinterpret_cast<float4 *>(i0 + grp < nlong ? part : Y);
            out[(uint64_t)cur.dst * (EG_PPR_LANES / 4) + sl] = acc;
        }
        cur = nxt;
    }
}

// Rows in parts: a warp per row adds its part sums, group g the g-th quarter
// of them in order with EG_PPR_FIXUP in flight, then the quarters in order.
// (A hub has thousands of parts: one load per step made their chain of
// latencies the kernel: undirected RMAT-20 64 us a sweep, now 8.)
#define EG_PPR_FIXUP 8
__global__ void __launch_bounds__(256) k_ppr_fixup(const uint4 *__restrict__ multi, uint32_t nmulti,
                                                   const float *__restrict__ part, float *__restrict__ Y) {
    const uint32_t lane = threadIdx.x & 31, grp = lane >> 3, sl = lane & 7;
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= nmulti) return;
    const uint4 r = multi[t];  // row, first part, parts
    const uint32_t per = (r.z + 3) >> 2;
    const uint32_t k0 = r.y + min(grp * per, r.z), k1 = r.y + min((grp + 1) * per, r.z);
    const float4 *__restrict__ P4 = reinterpret_cast<const float4 *>(part) + sl;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t k = k0; k < k1; k += EG_PPR_FIXUP) {
        float4 x[EG_PPR_FIXUP];
#pragma unroll
        for (uint32_t i = 0; i < EG_PPR_FIXUP; i++)
            if (k + i < k1) x[i] = __ldcg(P4 + (uint64_t)(k + i) * (EG_PPR_LANES / 4));
        float4 s = x[0];
#pragma unroll
        for (uint32_t i = 1; i < EG_PPR_FIXUP; i++)
            if (k + i < k1) s = eg_f4add(s, x[i]);
        acc = eg_f4add(acc, s);
    }
    float4 tot = eg_f4shfl(EG_FULL_MASK, acc, (int)sl);
#pragma unroll
    for (int g = 1; g < 4; g++) tot = eg_f4add(tot, eg_f4shfl(EG_FULL_MASK, acc, (int)(g * 8 + sl)));
    if (grp == 0) reinterpret_cast<float4 *>(Y)[(uint64_t)r.x * (EG_PPR_LANES / 4) + sl] = tot;
}

// Rows without in-edges sum to zero.  A lane tests one vertex (coalesced row
// pointers), the warp then writes the rows found.
__global__ void k_ppr_empty(const uint32_t *__restrict__ ptr, uint32_t n, float *__restrict__ Y) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint64_t v0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); v0 < n; v0 += stride) {
        const uint64_t v = v0 + lane;
        uint32_t found = __ballot_sync(EG_FULL_MASK, v < n && ptr[v] == ptr[v + 1]);
        while (found) {
            const uint32_t i = (uint32_t)__ffs(found) - 1;
            found &= found - 1;
            Y[(v0 + i) * EG_PPR_LANES + lane] = 0.f;
        }
    }
}

// Teleport plus returned dangling mass at the seeds: Y[s][q] += c_q / d so that
// d * Y carries (1 - d + d * dangling_q) / nseeds_q at every seed occurrence.
// Query q's seeds are seeds[sbeg[q] .. send[q]).  With `ptr` the rows without
// in-edges are zeroed only before the first sweep: a seed among them starts
// from zero here.
__global__ void k_ppr_seeds(const uint32_t *__restrict__ seeds, const uint32_t *__restrict__ sbeg,
                            const uint32_t *__restrict__ send, int nq, const PprQ *__restrict__ qs, float d,
                            float *__restrict__ Y, const uint32_t *__restrict__ ptr = nullptr) {
    const int q = threadIdx.x;
    if (q >= nq || !qs[q].active || qs[q].done) return;
    const float c = (float)(((1.0 - (double)d) + (double)d * qs[q].dangling) / ((double)qs[q].nseeds * (double)d));
    if (ptr)
        for (uint32_t i = sbeg[q]; i < send[q]; i++) {
            const uint32_t s = seeds[i];
            if (ptr[s] == ptr[s + 1]) Y[(uint64_t)s * EG_PPR_LANES + q] = 0.f;
        }
    for (uint32_t i = sbeg[q]; i < send[q]; i++) Y[(uint64_t)seeds[i] * EG_PPR_LANES + q] += c;
}

// R = d * Y, X = R / deg; per-block FP64 partials of |R - R_old| and of the
// mass on out-degree-0 vertices, per query.  Bound by HBM (four 128-byte rows
// per vertex): lane s of a group of 8 holds queries 4s .. 4s+3, so a warp has
// four rows of Y and R in flight (one before: 1 M vertices 278 us, now 105, the
// rows alone take 81 at the copy rate; two rows per group 126, four 112).  A finished or unused query keeps its R, and its
// X is written as the same R / deg again; groups of four such queries are
// skipped.
__global__ void __launch_bounds__(256) k_ppr_finish(const float *__restrict__ Y, const uint32_t *__restrict__ deg,
                                                    uint32_t n, float d, const PprQ *__restrict__ qs,
                                                    float *__restrict__ R, float *__restrict__ X,
                                                    double2 *__restrict__ part) {
    __shared__ double2 s_part[8][EG_PPR_LANES];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane >> 3, sl = lane & 7;
    bool live[4];
#pragma unroll
    for (int j = 0; j < 4; j++) live[j] = qs[4 * sl + j].active && !qs[4 * sl + j].done;
    eg_red2 acc[4];  // fp32 TwoSum pairs per query, widened once (FP64 issues slowly)
    if (live[0] | live[1] | live[2] | live[3]) {
        const float4 *__restrict__ Y4 = reinterpret_cast<const float4 *>(Y);
        float4 *R4 = reinterpret_cast<float4 *>(R), *X4 = reinterpret_cast<float4 *>(X);
        const uint64_t step = ((uint64_t)gridDim.x * blockDim.x) >> 3;  // groups of the grid
        for (uint64_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; v < n; v += step) {
            const uint64_t at = v * (EG_PPR_LANES / 4) + sl;
            const float4 y = __ldcs(Y4 + at), o = __ldcs(R4 + at);
            const uint32_t dv = __ldg(deg + v);
            const float yy[4] = {y.x, y.y, y.z, y.w}, oo[4] = {o.x, o.y, o.z, o.w};
            float r[4], x[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                r[j] = live[j] ? d * yy[j] : oo[j];
                x[j] = dv ? __fdiv_rn(r[j], (float)dv) : 0.f;
                acc[j].add(make_float2(fabsf(r[j] - oo[j]), dv ? 0.f : r[j]));
            }
            __stcs(R4 + at, make_float4(r[0], r[1], r[2], r[3]));
            X4[at] = make_float4(x[0], x[1], x[2], x[3]);
        }
    }
    // the four groups' pairs are merged as fp32 triples, then widened
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const eg_sum2 sum(acc[j]);  // groups 0 and 1 keep the first sum, 2 and 3 the second
        eg_sum3 mine = grp < 2 ? sum.a : sum.b;
        mine.add(eg_shfl_xor(grp < 2 ? sum.b : sum.a, 16));
        mine.add(eg_shfl_xor(mine, 8));
        const double w = mine.wide();
        if (grp == 0) s_part[warp][4 * sl + j].x = w;
        if (grp == 2) s_part[warp][4 * sl + j].y = w;
    }
    __syncthreads();
    if (warp == 0) {
        double2 s = make_double2(0.0, 0.0);
        for (int w = 0; w < 8; w++) {
            s.x += s_part[w][lane].x;
            s.y += s_part[w][lane].y;
        }
        part[(uint64_t)blockIdx.x * EG_PPR_LANES + lane] = s;
    }
}

// Per query: fixed-order FP64 sum of the block partials, stop test.  One CTA
// per query: FP64 adds issue so slowly here that one SM's worth of them was
// most of the kernel (16 us; one thread per query 61; now 4.4).
__global__ void __launch_bounds__(128) k_ppr_reduce(const double2 *__restrict__ part, uint32_t nblocks, PprQ *qs,
                                                    int count_iter) {
    __shared__ double2 s_sum[4];
    const uint32_t q = blockIdx.x;
    PprQ &s = qs[q];
    if (!s.active || s.done) return;
    double2 a = make_double2(0.0, 0.0);
#pragma unroll 4
    for (uint32_t b = threadIdx.x; b < nblocks; b += 128) {
        const double2 p = part[(uint64_t)b * EG_PPR_LANES + q];
        a.x += p.x;
        a.y += p.y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a.x += __shfl_down_sync(EG_FULL_MASK, a.x, o);
        a.y += __shfl_down_sync(EG_FULL_MASK, a.y, o);
    }
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = a;
    __syncthreads();  // every thread has tested s.done before it is set
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 4; w++) {
        a.x += s_sum[w].x;
        a.y += s_sum[w].y;
    }
    s.dangling = a.y;
    if (count_iter) {
        s.residual = a.x;
        s.iters += 1;
        if (a.x < (double)s.tol || s.iters >= s.max_iters) s.done = 1;
    }
}

// Zero the columns of the lanes in `mask` (every lane: mask = ~0).
__global__ void k_ppr_init(uint32_t n, uint32_t mask, float *R, float *X) {
    const uint64_t total = (uint64_t)n * EG_PPR_LANES;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        if (!((mask >> (i & 31)) & 1u)) continue;
        R[i] = 0.f;
        X[i] = 0.f;
    }
}
// Lanes in `mask` start from R = t: their columns must be zero on entry.
__global__ void k_ppr_init_seeds(const uint32_t *__restrict__ seeds, const uint32_t *__restrict__ sbeg,
                                 const uint32_t *__restrict__ send, uint32_t mask, const PprQ *qs,
                                 const uint32_t *__restrict__ deg, float *R, float *X) {
    const int q = threadIdx.x;
    if (q >= EG_PPR_LANES || !((mask >> q) & 1u) || !qs[q].active) return;
    const float w = 1.0f / (float)qs[q].nseeds;
    for (uint32_t i = sbeg[q]; i < send[q]; i++) R[(uint64_t)seeds[i] * EG_PPR_LANES + q] += w;
    for (uint32_t i = sbeg[q]; i < send[q]; i++) {
        const uint32_t s = seeds[i];
        const uint32_t dv = deg[s];
        X[(uint64_t)s * EG_PPR_LANES + q] = dv ? __fdiv_rn(R[(uint64_t)s * EG_PPR_LANES + q], (float)dv) : 0.f;
    }
}
__global__ void k_ppr_init_dangling(const uint32_t *__restrict__ seeds, const uint32_t *__restrict__ sbeg,
                                    const uint32_t *__restrict__ send, uint32_t mask,
                                    const uint32_t *__restrict__ deg, const float *R, PprQ *qs) {
    const int q = threadIdx.x;
    if (q >= EG_PPR_LANES || !((mask >> q) & 1u) || !qs[q].active) return;
    double dang = 0.0;
    for (uint32_t i = sbeg[q]; i < send[q]; i++) {
        const uint32_t s = seeds[i];
        bool first = true;  // count each distinct seed once
        for (uint32_t j = sbeg[q]; j < i; j++) first &= seeds[j] != s;
        if (first && deg[s] == 0) dang += (double)R[(uint64_t)s * EG_PPR_LANES + q];
    }
    qs[q].dangling = dang;
}

// out[q][v] = R[v][q] for q < nq: 32 x 32 tiles through shared memory.
__global__ void __launch_bounds__(256) k_ppr_extract(const float *__restrict__ R, uint32_t n, int nq,
                                                     float *__restrict__ out) {
    __shared__ float tile[32][EG_PPR_LANES + 1];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t v0 = (uint64_t)blockIdx.x * 32; v0 < n; v0 += (uint64_t)gridDim.x * 32) {
        for (uint32_t i = warp; i < 32; i += 8)
            if (v0 + i < n) tile[i][lane] = __ldcs(R + (v0 + i) * EG_PPR_LANES + lane);
        __syncthreads();
        for (uint32_t q = warp; q < (uint32_t)nq; q += 8)
            if (v0 + lane < n) out[(uint64_t)q * n + v0 + lane] = tile[lane][q];
        __syncthreads();
    }
}

}  // namespace
