// Single-source direction-optimising BFS as one cooperative launch: the level
// loop with grid barriers in place of a launch (or a host round trip) per
// step.
//
// A level is a push (the frontier listed with the running sum of its list
// lengths, every warp an equal share of the edges, hubs included) or a pull
// (every unvisited vertex looks for a parent in the frontier bitmap).  What a
// level reached is visited & ~prev, prev being the bitmap from before it, so
// that a push has one bitmap to claim in; the words are turned into a list or
// a frontier bitmap between levels, as the next direction needs.  Reads of
// words that other SMs write go through L1 where an old value is harmless (a
// visited bit missed is settled by the claim's atomicOr): every barrier makes
// the writes before it visible.
// Runs of small push levels go through one CTA while the others wait at a
// barrier (bfsl_small).
//
// What bounds it: on small graphs the barriers (1.2 us each on a part-filled
// grid, 4 .. 5 us with 304 CTAs) and one chain of dependent loads per step, on
// large ones the chain of a pull (visited, first, frontier word, in-list,
// frontier word).  Against a launch and a readback per level, call times:
// RMAT n = 5003, m = 80K 178 -> 80 us, n = 186K, m = 4.4M 205 -> 117 us,
// uniform n = 3M, m = 40M 450 -> 260 us, RMAT n = 16.8M, m = 537M 517 -> 385 us.
// 2 CTAs of 512 threads per SM: 3 take 372 us on the last, but 135 and 296 us
// on the two before it (spills, and barriers of more CTAs).
#pragma once
#include <cooperative_groups.h>

#include "eg_frontier.cuh"
#include "eg_internal.cuh"

#define EG_BFSL_T 512      // threads per CTA
#define EG_BFSL_B 2        // CTAs per SM
#define EG_BFSL_STEP 4     // places per lane in flight in a push
// Entries and vertices per CTA below a full grid.  The vertices count for the
// start values and the passes over the bitmaps: n = 16.8 M with 4 K entries,
// grid by the entries alone (3 CTAs) 1456 us, by both 59.
#define EG_BFSL_SHARE 4096u
#define EG_BFSL_ALONE 8    // 16-byte steps of a pull's list that one lane takes
#define EG_BFSL_SMALL 1024u  // edges of a push that one CTA takes alone
#define EG_NO_VERTEX 0xffffffffu

namespace {

struct BfsLoopState {
    unsigned long long deg[3];  // out-degree sum of the level reached: level i in set i % 3
    unsigned long long sel[2];  // list between levels: vertices << 32 | edges
    uint32_t count[3];          // vertices of the level reached
    uint32_t levels, pull_levels, err;
    unsigned long long reached, traversed;
    // what consecutive small levels left behind (bfsl_small)
    uint32_t s_count, s_levels;
    unsigned long long s_deg, s_reached, s_traversed;
};

struct BfsLoop {
    const uint32_t *ptr, *col, *iptr, *icol, *first, *noin, *deg;  // iptr NULL: push only
    uint32_t n, nw, root;
    int dirmode;
    double threshold;
    unsigned long long whole;  // the threshold, rounded down (bfsl_small)
    int32_t *level, *parent;
    uint32_t *visited, *prev, *bm[2];
    uint4 *queue;
    BfsLoopState *st;
};

struct BfsTally {
    uint32_t count;
    unsigned long long deg;
};

// The CTA's tally into a level's counters.
__device__ __forceinline__ void bfsl_add(BfsTally t, uint32_t *count, unsigned long long *deg) {
    __shared__ uint32_t s_count[EG_BFSL_T / 32];
    __shared__ unsigned long long s_deg[EG_BFSL_T / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        t.count += __shfl_down_sync(EG_FULL_MASK, t.count, o);
        t.deg += __shfl_down_sync(EG_FULL_MASK, t.deg, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_count[threadIdx.x >> 5] = t.count;
        s_deg[threadIdx.x >> 5] = t.deg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < EG_BFSL_T / 32; w++) {
            t.count += s_count[w];
            t.deg += s_deg[w];
        }
        if (t.count) {
            atomicAdd(count, t.count);
            atomicAdd(deg, t.deg);
        }
    }
}

// Shared memory of a CTA: a pull's lists and words, or the frontier of
// bfsl_small.  13 KB with the rest: two CTAs leave 196 KB of the SM to L1, which
// the pulls read their bitmaps through (25 KB: 164, pull-only searches of uniform
// n = 1M, m = 16M 297 -> 377 us).
union BfsSmem {
    struct {
        uint32_t list[EG_BFSL_T / 32][160];
        uint32_t found[EG_BFSL_T / 32][4];
    } pull;
    struct {
        uint2 q[EG_BFSL_SMALL];  // list start, length; from the level's scan on: start - place, first place
        uint32_t v[EG_BFSL_SMALL];
        uint32_t n[3], e[3], warp[EG_BFSL_T / 32];
    } small;
};

__device__ __forceinline__ bool bfsl_wants_pull(const BfsLoop &a, uint32_t count, unsigned long long fdeg) {
    return a.dirmode == EG_BFS_PULL_ONLY ||
           (a.dirmode == EG_BFS_AUTO && count + fdeg > a.whole);
}

// Push levels of at most EG_BFSL_SMALL edges, one after another in CTA 0 until
// the frontier is empty, larger, or one for a pull, the frontier in shared
// memory and block barriers between levels.  A level is one chain of three
// loads (entry, claim, row); by the whole grid it takes a list pass and two grid
// barriers.  A level of a path of 20,000 / 300,000 vertices: 6.1 / 7.2 us by the
// grid, now 1.4 / 2.1; a search of a 200 x 200 mesh 3.1 -> 1.0 ms, 1000 x 1000
// 22.4 -> 18.5.  A call of its own, and with whole-number compares, so that the
// other directions keep their registers (RMAT n = 16.8M, m = 537M: 430 us a
// search without this, 432 so, 438 inlined).
template <bool PARENT>
__device__ __noinline__ void bfsl_small(const BfsLoop &a, unsigned long long sel, uint32_t it, BfsSmem &sm) {
    static_assert(EG_BFSL_SMALL == 2 * EG_BFSL_T, "two edges, and two entries, per thread");
    auto &m = sm.small;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t cnt = (uint32_t)(sel >> 32), E = (uint32_t)sel, levels = 0, slot = 0;
    unsigned long long reached = 0, traversed = 0;
    for (uint32_t i = tid; i < cnt; i += EG_BFSL_T) {  // the list comes with its places
        const uint4 q = __ldcg(a.queue + i);
        m.q[i] = make_uint2(q.y, q.x);
        m.v[i] = q.z;
    }
    if (tid < 3) m.n[tid] = m.e[tid] = 0;
    __syncthreads();
    for (;;) {
        // up to 32 vertices: an entry per lane, every warp alike
        uint2 mine = make_uint2(0u, 0xffffffffu);
        if (cnt <= 32 && lane < cnt) mine = m.q[lane];
        if (cnt <= 32 && levels) {
            const uint32_t len = lane < cnt ? mine.y : 0u;
            uint32_t x = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(EG_FULL_MASK, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            if (lane < cnt) mine = make_uint2(mine.x - (x - len), x - len);
        }
        const int32_t next_level = (int32_t)(it + levels) + 2;
        uint32_t at[2], u[2];
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t x = tid + EG_BFSL_T * j;
            if (warp * 32 + EG_BFSL_T * j >= E) break;
            uint32_t o = 0, add;  // the last entry that begins at or before place x
            if (cnt <= 32) {
#pragma unroll
                for (uint32_t s = 16; s > 0; s >>= 1)
                    if (__shfl_sync(EG_FULL_MASK, mine.y, o + s) <= x) o += s;
                add = __shfl_sync(EG_FULL_MASK, mine.x, o);
            } else {
                for (uint32_t hi = cnt; hi - o > 1;) {
                    const uint32_t mid = (o + hi) >> 1;
                    if (m.q[mid].y <= x) o = mid;
                    else hi = mid;
                }
                add = m.q[o].x;
            }
            at[j] = x + add;
            u[j] = PARENT ? m.v[o] : 0u;
        }
        __syncthreads();  // the frontier is read: the next one takes its place
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t x = tid + EG_BFSL_T * j;
            if (warp * 32 + EG_BFSL_T * j >= E) break;
            uint32_t v = 0, old = EG_FULL_MASK, bit = 0, start = 0, len = 0;
            if (x < E) {
                v = __ldg(a.col + at[j]);
                bit = 1u << (v & 31);
                old = atomicOr(a.visited + (v >> 5), bit);
            }
            const bool claimed = !(old & bit) && x < E;
            if (claimed) {
                start = __ldg(a.ptr + v);
                len = __ldg(a.ptr + v + 1) - start;
                a.level[v] = next_level;
                if (PARENT) a.parent[v] = (int32_t)u[j];
            }
            const uint32_t ball = __ballot_sync(EG_FULL_MASK, claimed);
            if (!ball) continue;
            const uint32_t sum = __reduce_add_sync(EG_FULL_MASK, len);  // < 2^32 over all vertices
            uint32_t place = 0;
            if (lane == 0) {
                place = atomicAdd(&m.n[slot], (uint32_t)__popc(ball));
                atomicAdd(&m.e[slot], sum);
            }
            place = __shfl_sync(EG_FULL_MASK, place, 0) + __popc(ball & eg_lanemask_lt());
            if (claimed) {
                m.q[place] = make_uint2(start, len);
                m.v[place] = v;
            }
        }
        const uint32_t nslot = slot == 2 ? 0 : slot + 1;
        if (tid == 0) m.n[nslot] = m.e[nslot] = 0;  // read before the last barrier, used after the next
        __syncthreads();
        cnt = m.n[slot];
        E = m.e[slot];
        slot = nslot;
        levels++;
        reached += cnt;
        traversed += E;
        if (!cnt || E > EG_BFSL_SMALL || bfsl_wants_pull(a, cnt, E) || it + levels > a.n) break;
        // the frontier goes on here: visited & ~prev is to be what comes after it
        for (uint32_t i = tid; i < cnt; i += EG_BFSL_T) {
            const uint32_t v = m.v[i];
            atomicOr(a.prev + (v >> 5), 1u << (v & 31));
        }
        if (cnt > 32) {  // places: two entries per thread
            const uint32_t i = 2 * tid;
            const uint2 q0 = i < cnt ? m.q[i] : make_uint2(0u, 0u), q1 = i + 1 < cnt ? m.q[i + 1] : make_uint2(0u, 0u);
            const uint32_t s = q0.y + q1.y;
            uint32_t x = s;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(EG_FULL_MASK, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            if (lane == 31) m.warp[warp] = x;
            __syncthreads();
            uint32_t off = x - s;
            for (uint32_t w = 0; w < warp; w++) off += m.warp[w];
            if (i < cnt) m.q[i] = make_uint2(q0.x - off, off);
            if (i + 1 < cnt) m.q[i + 1] = make_uint2(q1.x - (off + q0.y), off + q0.y);
            __syncthreads();
        }
    }
    if (tid == 0) {
        a.st->s_count = cnt;
        a.st->s_levels = levels;
        a.st->s_deg = E;
        a.st->s_reached = reached;
        a.st->s_traversed = traversed;
    }
}

template <bool PARENT>
__device__ __forceinline__ BfsTally bfsl_push(const BfsLoop &a, unsigned long long sel, int32_t next_level) {
    BfsTally tally = {0u, 0ull};
    const uint32_t cnt = (uint32_t)(sel >> 32), E = (uint32_t)sel;
    const uint32_t lane = threadIdx.x & 31, le = eg_lanemask_lt() | (1u << lane);
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t per = (uint32_t)(((uint64_t)E + warps - 1) / warps);
    per = per < 64u ? 64u : (per + 31u) & ~31u;
    const uint64_t begin = (uint64_t)wid * per;
    if (begin >= E) return tally;
    uint32_t p = (uint32_t)begin;
    const uint32_t end = E - p > per ? p + per : E;
    uint32_t i0 = eg_list_find(&a.queue[0].x, 4u, cnt, p);
    for (; p < end; i0 += 32) {
        uint4 q = make_uint4(0xffffffffu, 0u, 0u, 0u);
        if (i0 + lane < cnt) q = __ldcg(a.queue + i0 + lane);
        const uint32_t wend = i0 + 32 < cnt ? __ldcg(&a.queue[i0 + 32].x) : E;
        const uint32_t stop = wend < end ? wend : end;
        for (; p < stop; p = stop - p > 32 * EG_BFSL_STEP ? p + 32 * EG_BFSL_STEP : stop) {
            uint32_t v[EG_BFSL_STEP], u[EG_BFSL_STEP], word[EG_BFSL_STEP];
            bool on[EG_BFSL_STEP];
#pragma unroll
            for (int k = 0; k < EG_BFSL_STEP; k++) {
                const uint32_t x0 = p + 32 * k;
                const uint32_t starts = __reduce_or_sync(EG_FULL_MASK, q.x - x0 < 32u ? 1u << (q.x - x0) : 0u);
                const uint32_t o = __popc(__ballot_sync(EG_FULL_MASK, q.x < x0)) - 1 + __popc(starts & le);
                const uint32_t at = x0 + lane + __shfl_sync(EG_FULL_MASK, q.y, o);
                if (PARENT) u[k] = __shfl_sync(EG_FULL_MASK, q.z, o);
                on[k] = stop - p > 32u * k + lane;
                v[k] = on[k] ? __ldg(a.col + at) : 0u;
            }
#pragma unroll
            for (int k = 0; k < EG_BFSL_STEP; k++) word[k] = on[k] ? __ldca(a.visited + (v[k] >> 5)) : EG_FULL_MASK;
#pragma unroll
            for (int k = 0; k < EG_BFSL_STEP; k++) {
                const uint32_t bit = 1u << (v[k] & 31);
                if (!(word[k] & bit)) word[k] = atomicOr(a.visited + (v[k] >> 5), bit);
                else word[k] = EG_FULL_MASK;
            }
#pragma unroll
            for (int k = 0; k < EG_BFSL_STEP; k++) {
                if (word[k] & (1u << (v[k] & 31))) continue;
                a.level[v[k]] = next_level;
                if (PARENT) a.parent[v[k]] = (int32_t)u[k];
                tally.count++;
                tally.deg += __ldg(a.deg + v[k]);
            }
        }
    }
    return tally;
}

// The first of list entries p .. p + 3 within [b, e) that is in the frontier
// (the array's end is padded).
__device__ __forceinline__ uint32_t bfsl_parent(const uint32_t *__restrict__ icol, const uint32_t *cur, uint32_t b,
                                                uint32_t e, uint32_t p) {
    const uint4 c4 = __ldg(reinterpret_cast<const uint4 *>(icol + p));
    const uint32_t c[4] = {c4.x, c4.y, c4.z, c4.w};
    uint32_t x[4], u = EG_NO_VERTEX;
#pragma unroll
    for (int j = 0; j < 4; j++) x[j] = p + j >= b && p + j < e ? __ldca(cur + (c[j] >> 5)) : 0u;
#pragma unroll
    for (int j = 3; j >= 0; j--)
        if ((x[j] >> (c[j] & 31)) & 1u) u = c[j];
    return u;
}

// The in-list of vertex t (EG_NO_VERTEX: none) against the frontier, one vertex
// per lane, four entries per step; a list that is longer than EG_BFSL_ALONE
// steps goes on 128 entries at a time.  Whole warps.
__device__ __forceinline__ uint32_t bfsl_scan(const BfsLoop &a, const uint32_t *cur, uint32_t t) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t u = EG_NO_VERTEX, p = 0, b = 0, e = 0, left = 0;  // left: entries from p to e
    if (t != EG_NO_VERTEX) {
        b = __ldg(a.iptr + t);
        e = __ldg(a.iptr + t + 1);
        p = b & ~3u;
        left = e - p;
    }
    for (int k = 0; k < EG_BFSL_ALONE && left && u == EG_NO_VERTEX; k++, p += 4) {
        u = bfsl_parent(a.icol, cur, b, e, p);
        left = left > 4 ? left - 4 : 0;
    }
    for (uint32_t rest = __ballot_sync(EG_FULL_MASK, left && u == EG_NO_VERTEX); rest; rest &= rest - 1) {
        const int l = __ffs(rest) - 1;
        const uint32_t at = __shfl_sync(EG_FULL_MASK, p, l), len = __shfl_sync(EG_FULL_MASK, left, l);
        uint32_t has = 0, w = EG_NO_VERTEX;
        for (uint32_t o = 0; !has; o += 128) {
            if (4 * lane < len - o) w = bfsl_parent(a.icol, cur, at, at + len, at + o + 4 * lane);
            has = __ballot_sync(EG_FULL_MASK, w != EG_NO_VERTEX);
            if (len - o <= 128) break;
        }
        if (has) w = __shfl_sync(EG_FULL_MASK, w, __ffs(has) - 1);
        if (has && lane == (uint32_t)l) u = w;
    }
    return u;
}

// A warp takes 4 bitmap words (128 vertices) per turn, 4 vertices per lane;
// small turns keep the warps' shares even (32 words per turn: 412 us instead of
// 260 on the uniform graph above).  Each unvisited vertex first tests
// its likely parent (first[]); the ones left over are collected in shared
// memory and scan their in-lists 32 at a time, the newest first, so that every
// lane has a list and most finds fall into the words of the turn at hand
// (scanned turn by turn: 412 us instead of 385 on the largest graph above).
template <bool PARENT>
__device__ __forceinline__ BfsTally bfsl_pull(const BfsLoop &a, const uint32_t *cur, uint32_t *next,
                                              int32_t next_level, BfsSmem &sm) {
    BfsTally tally = {0u, 0ull};
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, mine = lane >> 3, shift = 4 * (lane & 7);
    uint32_t *list = sm.pull.list[warp], *found = sm.pull.found[warp];
    const uint32_t step = ((gridDim.x * blockDim.x) >> 5) * 4;
    uint32_t w0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 4, held = 0;
    uint32_t ahead = w0 + mine < a.nw ? __ldcg(a.visited + w0 + mine) : EG_FULL_MASK;
    bool last = false;
    for (; !last; w0 += step) {
        last = w0 >= a.nw;  // one turn more for the rest of the list
        const uint32_t w = w0 + mine, vis = ahead;
        if (!last) ahead = w0 + step < a.nw && w + step < a.nw ? __ldcg(a.visited + w + step) : EG_FULL_MASK;
        uint32_t got = 0;
        const bool any = __any_sync(EG_FULL_MASK, vis != EG_FULL_MASK);
        if (any || last) {
            uint32_t bits = (~vis >> shift) & 15u, hit = 0;
            const uint32_t v = w0 * 32 + 4 * lane;
            if (lane < 4) found[lane] = 0;
            __syncwarp();
            if (bits) {
                const uint4 f4 = __ldg(reinterpret_cast<const uint4 *>(a.first + v));  // past n: no bits
                const uint32_t f[4] = {f4.x, f4.y, f4.z, f4.w};
                uint32_t x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (f[i] == EG_NO_VERTEX) bits &= ~(1u << i);  // no in-neighbours
                    x[i] = (bits >> i) & 1u ? __ldca(cur + (f[i] >> 5)) : 0u;
                }
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    if (!((bits >> i) & 1u) || !((x[i] >> (f[i] & 31)) & 1u)) continue;
                    hit |= 1u << i;
                    a.level[v + i] = next_level;
                    if (PARENT) a.parent[v + i] = (int32_t)f[i];
                    tally.count++;
                    tally.deg += __ldg(a.deg + v + i);
                }
                if (hit) atomicOr(&found[mine], hit << shift);
            }
            const uint32_t miss = bits & ~hit;
            uint32_t at = __popc(miss);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(EG_FULL_MASK, at, o);
                if (lane >= (uint32_t)o) at += y;
            }
            const uint32_t total = held + __shfl_sync(EG_FULL_MASK, at, 31);
            at += held - __popc(miss);
#pragma unroll
            for (int i = 0; i < 4; i++)
                if ((miss >> i) & 1u) list[at++] = v + i;
            __syncwarp();
            for (held = total; held >= 32 || (last && held);) {
                const uint32_t take = held < 32 ? held : 32;
                held -= take;
                const uint32_t t = lane < take ? list[held + lane] : EG_NO_VERTEX, u = bfsl_scan(a, cur, t);
                if (u == EG_NO_VERTEX) continue;
                a.level[t] = next_level;
                if (PARENT) a.parent[t] = (int32_t)u;
                tally.count++;
                tally.deg += __ldg(a.deg + t);
                const uint32_t k = (t >> 5) - w0, bit = 1u << (t & 31);
                if (k < 4) {
                    atomicOr(&found[k], bit);
                } else {  // of an earlier turn, whose words are written
                    atomicOr(next + (t >> 5), bit);
                    atomicOr(a.visited + (t >> 5), bit);
                }
            }
            __syncwarp();
            got = found[mine];
            __syncwarp();  // read by all before the next turn clears it
        }
        if (!last && !(lane & 7) && w < a.nw) {
            next[w] = got;
            a.prev[w] = vis;
            if (got) a.visited[w] = vis | got;
        }
    }
    return tally;
}

// visited & ~prev as a frontier bitmap.
__device__ __forceinline__ void bfsl_bitmap(const BfsLoop &a, uint32_t *bm) {
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < a.nw; w += gridDim.x * blockDim.x) {
        const uint32_t x = __ldcg(a.visited + w);
        bm[w] = x & ~a.prev[w];
        a.prev[w] = x;
    }
}

// Row starts ptr[v .. v + 4] (past the end: the buffer's padding).
__device__ __forceinline__ void bfsl_rows(const uint32_t *__restrict__ ptr, uint32_t v, bool on, uint32_t (&r)[5]) {
    const uint4 q = on ? __ldg(reinterpret_cast<const uint4 *>(ptr + v)) : make_uint4(0u, 0u, 0u, 0u);
    r[0] = q.x;
    r[1] = q.y;
    r[2] = q.z;
    r[3] = q.w;
    r[4] = on ? __ldg(ptr + v + 4) : 0u;
}

// visited & ~prev as a list for a push; vertices without out-edges are left out.
__device__ __forceinline__ void bfsl_list(const BfsLoop &a, unsigned long long *sel) {
    constexpr uint32_t NWARP = EG_BFSL_T / 32;
    __shared__ uint32_t s_cnt[NWARP], s_edges[NWARP];
    __shared__ unsigned long long s_base;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, shift = 4 * (lane & 7);
    // a warp takes up to 8 groups of 4 words (4 vertices per lane), fewer when
    // that leaves warps idle
    const uint32_t warps = gridDim.x * NWARP, all = (a.nw + 3) >> 2;
    uint32_t groups = (all + warps - 1) / warps;
    groups = groups > 8 ? 8 : groups;
    // uniform trip count per CTA
    for (uint32_t c0 = blockIdx.x * NWARP * groups * 4; c0 < a.nw; c0 += gridDim.x * NWARP * groups * 4) {
        const uint32_t w0 = c0 + warp * groups * 4;
        uint32_t keep = 0;                // bits 4g .. 4g + 3: the lane's listed vertices of group g
        uint32_t g_cnt = 0, g_edges = 0;  // of group `lane`
        for (uint32_t g = 0; g < groups; g++) {
            const uint32_t w = w0 + 4 * g + (lane >> 3);
            uint32_t x = 0, p = 0;
            if (w < a.nw) {
                x = __ldcg(a.visited + w);
                p = a.prev[w];
            }
            const uint32_t bits = ((x & ~p) >> shift) & 15u;
            if (!__any_sync(EG_FULL_MASK, x != p)) continue;
            if (!(lane & 7) && x != p) a.prev[w] = x;
            uint32_t r[5], k = 0, e = 0;
            bfsl_rows(a.ptr, (w0 + 4 * g) * 32 + 4 * lane, bits != 0u, r);
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (((bits >> i) & 1u) && r[i + 1] != r[i]) {
                    k |= 1u << i;
                    e += r[i + 1] - r[i];
                }
            keep |= k << (4 * g);
            const uint32_t c = __reduce_add_sync(EG_FULL_MASK, __popc(k));
            e = __reduce_add_sync(EG_FULL_MASK, e);
            if (lane == g) {
                g_cnt = c;
                g_edges = e;
            }
        }
        if (!__syncthreads_or(keep != 0u)) continue;
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
            for (uint32_t i = 0; i < NWARP; i++) {
                const uint32_t p = s_cnt[i], q = s_edges[i];
                s_cnt[i] = tc;
                s_edges[i] = te;
                tc += p;
                te += q;
            }
            // one word for both sums (m < 2^32), so that they keep the same order
            s_base = tc ? atomicAdd(sel, ((unsigned long long)tc << 32) | te) : 0ull;
        }
        __syncthreads();
        const uint32_t pc = (uint32_t)(s_base >> 32) + s_cnt[warp] + xc - g_cnt;
        const uint32_t pe = (uint32_t)s_base + s_edges[warp] + xe - g_edges;
        for (uint32_t g = 0; g < groups; g++) {
            const uint32_t bits = (keep >> (4 * g)) & 15u;
            if (!__any_sync(EG_FULL_MASK, bits != 0u)) continue;
            const uint32_t v = (w0 + 4 * g) * 32 + 4 * lane;
            uint32_t r[5], len = 0;
            bfsl_rows(a.ptr, v, bits != 0u, r);
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
                a.queue[at++] = make_uint4(off, r[i] - off, v + i, 0u);
                off += r[i + 1] - r[i];
            }
        }
        __syncthreads();  // s_cnt, s_edges and s_base are rewritten for the next words
    }
}

template <bool PARENT>
__global__ void __launch_bounds__(EG_BFSL_T, EG_BFSL_B) k_bfs_loop(const BfsLoop a) {
    __shared__ BfsSmem sm;
    auto grid = cooperative_groups::this_grid();
    const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    const uint32_t root = a.root;
    {  // levels and parents four vertices at a time (the arrays' ends are padded)
        const uint32_t nq = (uint32_t)(((uint64_t)a.n + 3) >> 2);
        for (uint32_t q = i0; q < nq; q += stride) {
            int4 l = make_int4(0, 0, 0, 0), p = make_int4(-1, -1, -1, -1);
            if (q == root >> 2) {
                reinterpret_cast<int *>(&l)[root & 3] = 1;
                reinterpret_cast<int *>(&p)[root & 3] = (int)root;
            }
            reinterpret_cast<int4 *>(a.level)[q] = l;
            if (PARENT) reinterpret_cast<int4 *>(a.parent)[q] = p;
        }
    }
    for (uint32_t w = i0; w < a.nw; w += stride) {
        const uint32_t bit = (root >> 5) == w ? 1u << (root & 31) : 0u;
        // vertices without in-neighbours can only be the root: the pulls skip them
        const uint32_t x = bit | (a.noin ? __ldg(a.noin + w) : 0u);
        a.visited[w] = x;
        a.prev[w] = x;
        a.bm[0][w] = bit;
    }
    const unsigned long long d0 = __ldg(a.deg + root);
    if (i0 == 0) {
        for (int i = 0; i < 3; i++) a.st->deg[i] = a.st->count[i] = 0;
        a.st->sel[0] = a.st->sel[1] = 0;
        a.queue[0] = make_uint4(0u, __ldg(a.ptr + root), root, 0u);
    }
    grid.sync();
    unsigned long long fdeg = d0, reached = 1, traversed = d0, sel = d0 ? (1ull << 32) | d0 : 0ull;
    uint32_t count = 1, pulls = 0, set = 0, it = 0, lists = 0;
    int cur = 0;
    auto wants_pull = [&]() {
        return a.dirmode == EG_BFS_PULL_ONLY ||
               (a.dirmode == EG_BFS_AUTO && (double)count + (double)fdeg > a.threshold);
    };
    bool pull = wants_pull(), over = false;
    for (;; it++) {
        const uint32_t nset = set == 2 ? 0 : set + 1;
        if (i0 == 0) {  // no CTA reads these any more, and none adds to them yet
            a.st->deg[nset] = 0;
            a.st->count[nset] = 0;
            a.st->sel[lists & 1] = 0;
        }
        const bool small = !pull && (uint32_t)(sel >> 32) <= EG_BFSL_SMALL && (uint32_t)sel <= EG_BFSL_SMALL;
        if (small) {
            if (blockIdx.x == 0) bfsl_small<PARENT>(a, sel, it, sm);
            grid.sync();
            count = __ldcg(&a.st->s_count);
            fdeg = __ldcg(&a.st->s_deg);
            reached += __ldcg(&a.st->s_reached);
            traversed += __ldcg(&a.st->s_traversed);
            it += __ldcg(&a.st->s_levels) - 1;
        } else {
            const int32_t next_level = (int32_t)it + 2;
            const BfsTally t = pull ? bfsl_pull<PARENT>(a, a.bm[cur], a.bm[cur ^ 1], next_level, sm)
                                    : bfsl_push<PARENT>(a, sel, next_level);
            __syncwarp();
            bfsl_add(t, &a.st->count[set], &a.st->deg[set]);
            grid.sync();
            count = __ldcg(&a.st->count[set]);
            fdeg = __ldcg(&a.st->deg[set]);
            reached += count;
            traversed += fdeg;
            pulls += pull;
            set = nset;
        }
        over = it > a.n;
        if (!count || over) break;
        const bool was = pull;
        pull = wants_pull();
        if (!pull) {
            bfsl_list(a, &a.st->sel[lists & 1]);
            grid.sync();
            sel = __ldcg(&a.st->sel[lists & 1]);
            lists++;
        } else if (was) {
            cur ^= 1;
        } else {
            bfsl_bitmap(a, a.bm[cur]);
            grid.sync();
        }
    }
    if (i0 == 0) {
        a.st->levels = it + 1;
        a.st->pull_levels = pulls;
        a.st->err = count && over;
        a.st->reached = reached;
        a.st->traversed = traversed;
    }
}

}  // namespace
