// PageRank on graphs small enough that launches, not entries, are the time:
// every iteration of a run in one cooperative launch.
//
// A kernel per step (row sums, row parts, empty rows, residual, reduction) is
// 5 launches and about 50 us per iteration whatever the size; here an
// iteration is one pass over a CTA's own rows and one grid barrier.  Each CTA
// owns an equal share of the rows with entries (a row weighing EG_PRS_ROW
// entries more than it has), keeps their columns in shared memory for the
// whole run, and (STAGE: up to EG_PRS_STAGE_N vertices) copies the contributions
// there every iteration, so that the gathers stay in the SM; above, they are
// gathered from L2 (L1 could hold the last iteration's).  A row is summed by one lane up to EG_PRS_LANE
// entries, by 8 lanes up to EG_PRS_GROUP, by a warp up to EG_PRS_WARP, else by
// the CTA; the order is fixed, so a run's bits are too.  The residual and the
// dangling mass are summed as fp32 triples and widened once:
// FP64 issues so slowly here that an FP64 pair per warp was half an iteration.
//
// Ten iterations (or to 1e-6), one call, before -> now: 1,250 vertices 354 ->
// 86 us; 10,007 and 240 K entries to 1e-6 816 -> 198; 40,170 and 2 M 412 ->
// 153; gathered from L2: 41,007 and 840 K 342 -> 120, 83,170 and 816 K to 1e-6
// 921 -> 554, 300,007 and 2 M 463 -> 378, but 1,000,007 and 4 M 522 -> 674 and
// 100,007 and 4.2 M 454 -> 459: hence the limits.
#pragma once
#include <cooperative_groups.h>

#include <type_traits>

#include "eg_internal.cuh"

#define EG_PRS_THREADS 1024
#define EG_PRS_STAGE_N 40960u       // contributions: 160 KB of the 227 KB
#define EG_PRS_STAGE_M (1u << 22)   // entries with staged contributions
#define EG_PRS_MAX_N (1u << 18)     // without
#define EG_PRS_MAX_M (1u << 21)
#define EG_PRS_ROW 8u
#define EG_PRS_LANE 8u
#define EG_PRS_GROUP 128u
#define EG_PRS_WARP 4096u
#define EG_PRS_MAX_LONG 64u
#define EG_PRS_SHARE 2048u          // entries per CTA below a full grid (and EG_PRS_THREADS vertices)

namespace {

struct PrSmall {
    const uint32_t *ptr, *col, *deg, *perm;
    uint32_t n, rows, m;  // rows [rows, n) have no entries
    uint32_t mult;
    int iterations, swap, dangling;
    float damping, prev_init;
    double base0, per_dangling, tol;  // base = base0 + per_dangling * dangling mass
    float *c0, *c1, *rank_p, *rank;
    eg_sum2 *part;  // two sets of one pair of sums per CTA
    eg_pr_dev *st;
    uint32_t cap;  // columns kept in shared memory
};

// Rows of [0, rows) that begin before x, a row being EG_PRS_ROW entries longer
// than it is (a whole warp).
__device__ __forceinline__ uint32_t prs_rows_below(const uint32_t *__restrict__ ptr, uint32_t rows, uint64_t x) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, len = rows;
    while (len) {
        const uint32_t s = (len + 31) >> 5, k = lane * s;
        const uint32_t c = (uint32_t)__popc(__ballot_sync(
            EG_FULL_MASK, k < len && (uint64_t)__ldg(ptr + lo + k) + (uint64_t)EG_PRS_ROW * (lo + k) < x));
        if (!c) break;
        const uint32_t past = (c - 1) * s + 1;  // that many are below
        lo += past;
        len = len - past < s - 1 ? len - past : s - 1;
    }
    return lo;
}

// The total of the CTAs' first (which 0) or second sums, in lane 0 of a warp,
// all of a lane's loads in flight up to 160 CTAs; past fp32's range in FP64.
__device__ __forceinline__ double prs_total(const eg_sum2 *part, uint32_t n, uint32_t which) {
    const uint32_t lane = threadIdx.x & 31;
    auto at = [&](uint32_t i) {
        const float *p = reinterpret_cast<const float *>(part + i) + 3 * which;
        eg_sum3 x;
        if (i < n) {
            x.s = __ldcg(p);
            x.c = __ldcg(p + 1);
            x.e = __ldcg(p + 2);
        }
        return x;
    };
    eg_sum3 sum;
    for (uint32_t i = lane; i - lane < n; i += 160) {
        eg_sum3 x[5];
#pragma unroll
        for (uint32_t k = 0; k < 5; k++) x[k] = at(i + 32 * k);
#pragma unroll
        for (uint32_t k = 0; k < 5; k++) sum.add(x[k]);
    }
    sum.add(eg_shfl_xor(sum, 16));
    sum = eg_half_sum(sum);
    if (__all_sync(EG_FULL_MASK, isfinite(sum.s))) return sum.wide();
    double t = 0.0;
    for (uint32_t i = lane; i < n; i += 32) t += at(i).wide();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(EG_FULL_MASK, t, o);
    return t;
}

// REDUCE: the residual and the dangling mass are wanted (a tolerance, or
// dangling mass spread).
template <bool REDUCE, bool STAGE>
__global__ void __launch_bounds__(EG_PRS_THREADS, 1) k_pr_small(const PrSmall a) {
    extern __shared__ __align__(16) unsigned char prs_raw[];
    __shared__ eg_sum2 s_sum[EG_PRS_THREADS / 32];
    __shared__ float s_part[EG_PRS_THREADS / 32];
    __shared__ uint32_t s_row[2], s_long[EG_PRS_MAX_LONG], s_nlong;
    __shared__ float s_base;
    __shared__ int s_done;
    auto grid = cooperative_groups::this_grid();
    float *s_c = reinterpret_cast<float *>(prs_raw);
    using Col = typename std::conditional<STAGE, uint16_t, uint32_t>::type;
    Col *s_col = reinterpret_cast<Col *>(prs_raw + (STAGE ? (a.n * 4ull + 15) & ~15ull : 0ull));
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x, b = blockIdx.x;
    if (warp < 2) {
        const uint32_t r = b + warp == G ? a.rows : prs_rows_below(a.ptr, a.rows, (uint64_t)(b + warp) * (a.m + (uint64_t)EG_PRS_ROW * a.rows) / G);
        if (lane == 0) s_row[warp] = r;
    }
    if (tid == 0) s_nlong = 0;
    __syncthreads();
    const uint32_t R0 = s_row[0], R1 = s_row[1], E0 = __ldg(a.ptr + R0), E1 = __ldg(a.ptr + R1);
    const uint32_t kept = E1 - E0 < a.cap ? E1 - E0 : a.cap;
    for (uint32_t e = tid; e < kept; e += EG_PRS_THREADS) s_col[e] = (Col)__ldg(a.col + E0 + e);
    // the rows for the whole CTA: at most m / (G * EG_PRS_WARP) + 1 of them
    for (uint32_t r = R0 + tid; r < R1; r += EG_PRS_THREADS)
        if (__ldg(a.ptr + r + 1) - __ldg(a.ptr + r) > EG_PRS_WARP) s_long[atomicAdd(&s_nlong, 1u)] = r;
    // the start vector, in equal shares of the vertices
    const uint32_t per = (a.n + G - 1) / G, v0 = b * per < a.n ? b * per : a.n, v1 = a.n - v0 < per ? a.n : v0 + per;
    eg_sum2 acc;
    for (uint32_t v = v0 + tid; v < v1; v += EG_PRS_THREADS) {
        const uint32_t d = __ldg(a.deg + v) * a.mult;
        __stcg(a.rank_p + v, a.prev_init);
        __stcg(a.c0 + v, d ? __fdiv_rn(a.prev_init, (float)d) : 0.f);
        acc.b.add(d ? 0.f : a.prev_init);
    }
    __syncthreads();
    if (tid == 0)  // in row order, so that the sums below keep one order
        for (uint32_t i = 1; i < s_nlong; i++)
            for (uint32_t j = i; j > 0 && s_long[j] < s_long[j - 1]; j--) {
                const uint32_t t = s_long[j];
                s_long[j] = s_long[j - 1];
                s_long[j - 1] = t;
            }
    if (REDUCE) eg_store_sum(eg_block_sum(acc, s_sum), a.part + b);
    const uint32_t eper = (a.n - a.rows + G - 1) / G;  // rows without entries, in equal shares
    const uint32_t x0 = a.n - a.rows > b * eper ? a.rows + b * eper : a.n, x1 = a.n - x0 < eper ? a.n : x0 + eper;
    for (int it = 0;; it++) {
        grid.sync();
        const bool odd = a.swap && (it & 1);
        const float *cin = odd ? a.c1 : a.c0;
        float *cout = odd ? a.c0 : a.c1;
        // the sums of the last pass, by every CTA alike: the next base, the stop test
        if (warp < 2) {
            // warp 0: the residual and the stop test, warp 1: the dangling mass and the base
            double t = 0.0;
            if (REDUCE) t = prs_total(a.part + (it & 1) * G, G, warp);
            if (lane == 0 && warp == 0) {
                s_done = it == a.iterations || (REDUCE && it && a.tol > 0.0 && t < a.tol);
                if (b == 0 && s_done) {
                    a.st->done = it < a.iterations;
                    a.st->iters = it;
                    a.st->residual = it ? t : 0.0;
                }
            } else if (lane == 0) {
                s_base = (float)(a.dangling ? a.base0 + a.per_dangling * t : a.base0);
                if (b == 0) {  // the last pass's stay
                    a.st->base = s_base;
                    a.st->dangling = t;
                }
            }
        } else if (STAGE && (it == 0 || a.swap)) {
            const uint32_t nq = a.n >> 2;
            for (uint32_t i = tid - 64; i < nq; i += EG_PRS_THREADS - 64)
                reinterpret_cast<float4 *>(s_c)[i] = __ldcg(reinterpret_cast<const float4 *>(cin) + i);
            if (tid - 64 < (a.n & 3)) s_c[4 * nq + tid - 64] = __ldcg(cin + 4 * nq + tid - 64);
        }
        __syncthreads();
        if (s_done) break;
        const float base = s_base;
        acc = eg_sum2();
        auto gather = [&](uint32_t e) -> float {
            const uint32_t i = e - E0;
            const uint32_t u = i < kept ? (uint32_t)s_col[i] : __ldg(a.col + e);
            return STAGE ? s_c[u] : __ldcg(cin + u);
        };
        // the row's last rank, for the residual: loaded before the row is summed
        auto last_rank = [&](uint32_t r) { return REDUCE && a.tol > 0.0 ? __ldcg(a.rank_p + r) : 0.f; };
        auto emit = [&](uint32_t r, float s, float old) {
            const float x = fmaf(a.damping, s, base);
            const uint32_t d = __ldg(a.deg + r) * a.mult;
            if (REDUCE) {
                acc.a.add(fabsf(x - old));
                acc.b.add(d ? 0.f : x);
            }
            __stcg(a.rank_p + r, x);
            if (a.swap) __stcg(cout + r, d ? __fdiv_rn(x, (float)d) : 0.f);
        };
        const uint32_t nlong = s_nlong;
        for (uint32_t i = 0; i < nlong; i++) {
            const uint32_t r = s_long[i], end = __ldg(a.ptr + r + 1);
            const float old = tid == 0 ? last_rank(r) : 0.f;
            float s = 0.f;
            for (uint32_t e = __ldg(a.ptr + r) + tid; e < end; e += 4 * EG_PRS_THREADS) {
                float x[4];
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) x[k] = e + k * EG_PRS_THREADS < end ? gather(e + k * EG_PRS_THREADS) : 0.f;
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) s += x[k];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(EG_FULL_MASK, s, o);
            if (lane == 0) s_part[warp] = s;
            __syncthreads();
            if (warp == 0) {
                s = s_part[lane];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(EG_FULL_MASK, s, o);
                if (lane == 0) emit(r, s, old);
            }
            __syncthreads();
        }
        for (uint32_t r = R0 + tid; r < R1; r += EG_PRS_THREADS) {
            const uint32_t e = __ldg(a.ptr + r), len = __ldg(a.ptr + r + 1) - e;
            if (len > EG_PRS_LANE) continue;
            const float old = last_rank(r);
            float x[EG_PRS_LANE], s = 0.f;
#pragma unroll
            for (uint32_t k = 0; k < EG_PRS_LANE; k++) x[k] = k < len ? gather(e + k) : 0.f;
#pragma unroll
            for (uint32_t k = 0; k < EG_PRS_LANE; k++) s += x[k];
            emit(r, s, old);
        }
        // a warp takes four rows at a time, 32 apart (neighbours have like
        // lengths): the ones for a warp in turn, then the others together
        const uint32_t sl = tid & 7, grp = lane >> 3;
        for (uint32_t r0 = R0 + warp; r0 < R1; r0 += EG_PRS_THREADS / 8) {
            const uint32_t r = r0 + 32 * grp;
            uint32_t e = 0, end = 0;
            if (r < R1) {
                e = __ldg(a.ptr + r);
                end = __ldg(a.ptr + r + 1);
            }
            const uint32_t len = end - e;
            if (!__any_sync(EG_FULL_MASK, len > EG_PRS_LANE)) continue;
            const float old = sl == 0 && len > EG_PRS_LANE && len <= EG_PRS_WARP ? last_rank(r) : 0.f;
            uint32_t wide = __ballot_sync(EG_FULL_MASK, sl == 0 && len > EG_PRS_GROUP && len <= EG_PRS_WARP);
            while (wide) {
                const int src = __ffs(wide) - 1;
                wide &= wide - 1;
                const uint32_t we = __shfl_sync(EG_FULL_MASK, e, src), wend = __shfl_sync(EG_FULL_MASK, end, src);
                float s = 0.f;
                for (uint32_t p = we + lane; p < wend; p += 128) {
                    float x[4];
#pragma unroll
                    for (uint32_t k = 0; k < 4; k++) x[k] = p + 32 * k < wend ? gather(p + 32 * k) : 0.f;
#pragma unroll
                    for (uint32_t k = 0; k < 4; k++) s += x[k];
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(EG_FULL_MASK, s, o);
                if ((int)lane == src) emit(r, s, old);
            }
            const bool mine = len > EG_PRS_LANE && len <= EG_PRS_GROUP;
            float s = 0.f;
            if (mine)
                for (e += sl; e < end; e += 32) {
                    float x[4];
#pragma unroll
                    for (uint32_t k = 0; k < 4; k++) x[k] = e + 8 * k < end ? gather(e + 8 * k) : 0.f;
#pragma unroll
                    for (uint32_t k = 0; k < 4; k++) s += x[k];
                }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(EG_FULL_MASK, s, o);
            if (mine && sl == 0) emit(r, s, old);
        }
        for (uint32_t r = x0 + tid; r < x1; r += EG_PRS_THREADS) emit(r, 0.f, last_rank(r));
        if (REDUCE) eg_store_sum(eg_block_sum(acc, s_sum), a.part + ((it + 1) & 1) * G + b);
    }
    for (uint32_t v = v0 + tid; v < v1; v += EG_PRS_THREADS) a.rank[v] = __ldcg(a.rank_p + __ldg(a.perm + v));
}

}  // namespace
