// Pull side of frontier SSSP: candidate labels over a row's in-edges, shared
// by the single-GPU sweep (sssp.cu) and the vertex-range shards (shard.cu).
//
// A sweep is bound like a PageRank iteration (pagerank.cu): one 32-byte L2
// sector per gathered label, at the rate that the L1 left beside shared
// memory allows.  So rows take their minimum straight from registers, by 1 to
// 8 lanes or a warp, and shared memory holds at most the hot-slot table.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "graph.cuh"
#include "sssp_core.cuh"

namespace hyt {
namespace ssp {

// In-edges of one task, addressed relative to its first edge.
struct InEdges {
    const uint32_t *src;    // source ids, hot ones tagged kHotTag | slot
    const uint32_t *w;      // weights in CSC order (NULL when unweighted), or packed words
    const uint32_t *s_hot;  // vertex ids of the hot slots (not with packed words)
    uint32_t bits;          // packed words: bits of the source id
    uint32_t inf;           // infinity label
};

// Lowest candidate label(u) + w over the edges b, b + kStep, ... below e, at
// most kN of them, all loaded before the first is used (`best` when none is
// lower); unreached sources give infinity or more.  A minimum does not mind an
// edge taken twice, so threads without an edge of their own repeat the row's
// last one (the same sector) in place of predicated loads: without packed words,
// u32 weights on R-MAT scale 24 in input order take 3.58 ms in place of 4.12 and
// f32 weights 5.95 in place of 6.06.  A row without edges gives an arbitrary
// result.
// kPacked: one word per edge, labels that cannot wrap (GraphImpl::
// in_pack_bits): a candidate is one add-and-min.  Half the instructions per edge
// of the general form, which streams ids and weights apart, maps hot slots and
// saturates: one source on R-MAT scale 24 took 2.38 ms in place of 2.83 (hub
// order) and 2.63 in place of 4.12 (input order; both with uneven tasks handed
// out one by one).
template <int kN, int kStep, int WK, bool kPacked, class Label>
__device__ __forceinline__ uint32_t edges_min(const InEdges &E, uint32_t b, uint32_t e, Label &&label, uint32_t best) {
    const uint32_t last = e > 0 ? e - 1 : 0u;
    uint32_t x[kN], du[kN];
    if constexpr (kPacked) {
        const uint32_t mask = (1u << E.bits) - 1u;
#pragma unroll
        for (int j = 0; j < kN; ++j) x[j] = dev::ld_stream(E.w + min(b + j * kStep, last));
#pragma unroll
        for (int j = 0; j < kN; ++j) du[j] = label(x[j] & mask);
#pragma unroll
        for (int j = 0; j < kN; ++j) best = __viaddmin_u32(du[j], x[j] >> E.bits, best);
    } else {
        uint32_t w[kN];
#pragma unroll
        for (int j = 0; j < kN; ++j) x[j] = dev::ld_stream(E.src + min(b + j * kStep, last));
#pragma unroll
        for (int j = 0; j < kN; ++j)
            if (x[j] & kHotTag) x[j] = E.s_hot[x[j] & ~kHotTag];
#pragma unroll
        for (int j = 0; j < kN; ++j) du[j] = label(x[j]);
#pragma unroll
        for (int j = 0; j < kN; ++j) w[j] = ssc::edge_weight<WK>(E.w, min(b + j * kStep, last));
#pragma unroll
        for (int j = 0; j < kN; ++j) {
            const uint32_t c = ssc::extend<WK>(du[j], w[j]);
            // a float infinity stays one by itself
            best = min(best, WK != HYT_WEIGHTS_F32 && du[j] == E.inf ? E.inf : c);
        }
    }
    return best;
}

// Lowest candidate over edges [b, e), by the whole warp; every lane returns it.
template <int WK, bool kPacked, class Label>
__device__ __forceinline__ uint32_t span_min(const InEdges &E, uint32_t b, uint32_t e, Label &&label, int lane) {
    constexpr int kN = 8;
    uint32_t best = E.inf;
    for (uint32_t at = b; at < e; at += 32 * kN) {
        if (e - at <= 16 * kN)  // a short last pass issues half of the slots
            best = edges_min<kN / 2, 32, WK, kPacked>(E, at + lane, e, label, best);
        else
            best = edges_min<kN, 32, WK, kPacked>(E, at + lane, e, label, best);
    }
    return __reduce_min_sync(0xffffffffu, best);
}

// Lowest candidates of the warp's 32 rows (lane l: edges [lo, hi)), kG lanes
// per row and 32 / kG rows a step; rows have at most kG * kN in-edges.
template <int kG, int kN, int WK, bool kPacked, class Label>
__device__ __forceinline__ uint32_t group_min(const InEdges &E, uint32_t lo, uint32_t hi, Label &&label, int lane) {
    constexpr int kRows = 32 / kG;
    uint32_t mine = E.inf;
    const uint32_t live = __ballot_sync(0xffffffffu, hi > lo);
    for (int step = 0; step < kG; ++step) {
        if (!((live >> (step * kRows)) & (kRows == 32 ? 0xFFFFFFFFu : (1u << (kRows % 32)) - 1u))) continue;
        const int owner = step * kRows + lane / kG;
        const uint32_t b = __shfl_sync(0xffffffffu, lo, owner) + (lane % kG);
        const uint32_t e = __shfl_sync(0xffffffffu, hi, owner);
        uint32_t best = edges_min<kN, kG, WK, kPacked>(E, b, e, label, E.inf);
#pragma unroll
        for (int o = 1; o < kG; o <<= 1) best = min(best, __shfl_xor_sync(0xffffffffu, best, o));
        const uint32_t t = __shfl_sync(0xffffffffu, best, (lane % kRows) * kG);
        if (lane / kRows == step) mine = t;
    }
    return hi > lo ? mine : E.inf;
}

constexpr uint32_t kWideRow = 64;  // rows with this many in-edges are taken by the whole warp

// Lowest candidate of each lane's row [lo, hi) (empty: infinity).  Rows of
// kWideRow or more in-edges one after another by the whole warp; the others by
// the smallest group of lanes that leaves each at most 8 edges of the largest
// (one round of loads per row).  Must be called by all 32 lanes.
template <int WK, bool kPacked, class Label>
__device__ __forceinline__ uint32_t rows_min(const InEdges &E, uint32_t lo, uint32_t hi, Label &&label, int lane) {
    const bool wide = hi - lo >= kWideRow;
    const uint32_t hs = wide ? lo : hi;  // group steps see a wide row as empty
    const uint32_t most = __reduce_max_sync(0xffffffffu, hs - lo);
    uint32_t best = E.inf;
    if (most > 32)
        best = group_min<8, 8, WK, kPacked>(E, lo, hs, label, lane);
    else if (most > 16)
        best = group_min<4, 8, WK, kPacked>(E, lo, hs, label, lane);
    else if (most > 8)
        best = group_min<2, 8, WK, kPacked>(E, lo, hs, label, lane);
    else if (most > 4)
        best = group_min<1, 8, WK, kPacked>(E, lo, hs, label, lane);
    else if (most > 2)
        best = group_min<1, 4, WK, kPacked>(E, lo, hs, label, lane);
    else if (most)
        best = group_min<1, 2, WK, kPacked>(E, lo, hs, label, lane);
    for (uint32_t big = __ballot_sync(0xffffffffu, wide); big; big &= big - 1) {
        const int r = __ffs(big) - 1;
        const uint32_t t = span_min<WK, kPacked>(E, __shfl_sync(0xffffffffu, lo, r), __shfl_sync(0xffffffffu, hi, r),
                                                 label, lane);
        if (lane == r) best = t;
    }
    return best;
}

}  // namespace ssp
}  // namespace hyt
