// Frontier building blocks shared by the single-source BFS and SSSP loops.
//
// eg_warp_lists  a warp walks the out-lists of its 32 lanes' vertices
//                together, 32 edges per step: an inclusive scan of the list
//                lengths gives each edge slot its owner lane by a 5-step
//                shuffle search, so every lane has an edge whatever the
//                degrees (one warp per vertex leaves most lanes idle on
//                low-degree frontiers).
// eg_list_find   the entry of a list with running sums that holds a place.
#pragma once
#include "eg_internal.cuh"

namespace {

// Lane i holds vertex u, list start b and length d (d = 0: nothing).  For
// every edge slot f(valid, owner_lane, owner_vertex, edge_index) is called
// by all 32 lanes together (so f may use warp collectives); edge_index is
// meaningful only where valid.
template <class F>
__device__ __forceinline__ void eg_warp_lists(uint32_t u, uint32_t b, uint32_t d, F &&f) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t inc = d;  // inclusive scan of the lengths
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(EG_FULL_MASK, inc, o);
        if (lane >= o) inc += y;
    }
    const uint32_t total = __shfl_sync(EG_FULL_MASK, inc, 31);
    const uint32_t exc = inc - d;
    for (uint32_t p0 = 0, left = total; left; p0 += 32, left = left > 32 ? left - 32 : 0) {
        const uint32_t x = p0 + lane;
        uint32_t lo = 0;  // owner of slot x: the first lane whose inclusive sum exceeds x
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1) {
            const uint32_t probe = __shfl_sync(EG_FULL_MASK, inc, lo + step - 1);
            if (probe <= x) lo += step;
        }
        const uint32_t ob = __shfl_sync(EG_FULL_MASK, b, lo);
        const uint32_t oe = __shfl_sync(EG_FULL_MASK, exc, lo);
        const uint32_t ou = __shfl_sync(EG_FULL_MASK, u, lo);
        const bool valid = lane < left;  // x may not fit 32 bits
        f(valid, lo, ou, valid ? ob + (x - oe) : 0u);
    }
}

// The list entry that holds place p: the last i with off[i * stride] <= p
// (off[0] = 0), found by a whole warp, 32 probes per step.
__device__ __forceinline__ uint32_t eg_list_find(const uint32_t *__restrict__ off, uint32_t stride, uint32_t cnt,
                                              uint32_t p) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t i0 = 0, len = cnt;
    while (len > 1) {
        const uint32_t s = (len + 31) >> 5, k = lane * s;
        const uint32_t b =
            __ballot_sync(EG_FULL_MASK, k < len && __ldcg(off + (uint64_t)(i0 + k) * stride) <= p);
        const uint32_t at = (31u - (uint32_t)__clz(b)) * s;  // bit 0 is set
        i0 += at;
        len = len - at < s ? len - at : s;
    }
    return i0;
}

}  // namespace
