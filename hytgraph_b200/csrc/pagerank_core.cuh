// Device building blocks of pull PageRank / personalized PageRank, shared
// by the single-query solver (pagerank.cu), the partitioned out-of-HBM
// solver and the batched multi-query engine (batch.cu): the per-row
// finalisation, the batched contribution gather, and the two task kinds
// (merge-path tile of short rows; chunk of a long row merged by its last
// arriving warp).  Semantics are described at the top of pagerank.cu.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "graph.cuh"

namespace hyt {
namespace prc {

#ifndef HYT_PR_WARP_ROW
#define HYT_PR_WARP_ROW 64
#endif
constexpr uint32_t kWarpRowDegree = HYT_PR_WARP_ROW;  // rows with this many in-edges are summed by a whole warp
static_assert(kWarpRowDegree <= 64, "8 lanes of 8 edges sum the other rows");

struct PRHeader {
    uint32_t iter;       // iterations completed
    uint32_t done;
    uint32_t converged;
    uint32_t error;      // 1: a bounded wait at a grid barrier ran out
    double last_residual;
};

// Fixed-order reduction of an iteration's residual and dangling mass.
// Every task owns a slot: tile k -> num_long + k, long row i -> i (written
// by the warp that finalizes the row) -- a plain store, nothing waits on it.
// After the iteration's tasks, pr_reduce_kernel sums each group of
// kSlotGroup slots in slot order (a fixed block tree), and its last block
// sums the group sums in group order and closes the iteration.  The result
// is the same for any grid, launch split or arrival order.  The counter
// only grows (each iteration adds the reduce grid), so it is cleared once
// per solve.
constexpr uint32_t kSlotGroup = 1024;

struct PRSlots {
    double2 *slot;          // [2 * num_slots] (residual, dangling); the persistent solver alternates halves
    double2 *group_sum;     // [num_groups]
    uint32_t *blocks_done;  // [4] reduce blocks finished, over the whole solve (persistent solver: barrier
                            // count), then the persistent solver's three task cursors
    uint32_t num_slots, num_groups;
};

// Arguments of a solve: kernel parameters, or an array in device memory (the
// launch-by-launch kernels' copy, the batch engine's slots).
struct PRArgs {
    const uint64_t *in_off;
    const uint32_t *in_src;
    const uint32_t *out_deg;
    const uint32_t *tile_start;
    const LongRow *long_rows;
    const uint2 *chunk_tasks;
    const uint32_t *hot_vertex;  // [num_hot] vertices cached in shared memory
    uint32_t num_hot;
    uint32_t tile_cost, chunk_edges;
    float *rank[2];
    float *contrib[2];
    float2 *partial;
    uint32_t *ticket;
    PRHeader *hdr;
    double *residual;        // [max_iter]
    double *dangling;        // [max_iter + 1]
    uint64_t num_tiles;
    uint32_t num_chunks;
    uint32_t V;
    float damping;
    float base;         // PR: (1-d)/n
    float tolerance;
    uint32_t max_iter;
    uint32_t source;    // PPR
    uint32_t personalized;
    PRSlots red;        // fixed-order residual / dangling reduction (single-query solver)
    const uint4 *tasks; // pull task descriptors
};

struct PRState {
    // per-iteration scalars
    float damping, base, teleport_scale;
    float dshare;  // PR: d * dangling / n
    float tele;    // PPR: (1-d) + d * dangling
    uint32_t source;
    bool personalized;
};

// Row r's next rank, contribution, L1 change and dangling share from its
// in-edge sum, given its current rank `old` and out-degree `od`.
__device__ __forceinline__ void finalize_row_with(const PRState &ps, uint32_t r, float sum, float old, uint32_t od,
                                                  float *nxt, float *cnxt, double &res, double &dang) {
    float nx;
    if (ps.personalized) {
        nx = __fmul_rn(ps.damping, sum);
        if (r == ps.source) nx = __fadd_rn(ps.tele, nx);
    } else {
        nx = __fadd_rn(ps.dshare, __fmul_rn(ps.damping, sum));
    }
    res += fabs(static_cast<double>(nx) - static_cast<double>(old));
    nxt[r] = nx;
    cnxt[r] = od ? __fdiv_rn(nx, static_cast<float>(od)) : 0.0f;
    if (od == 0) dang += static_cast<double>(nx);
}

__device__ __forceinline__ void finalize_row(const PRArgs &a, const PRState &ps, uint32_t r, float sum,
                                             const float *cur, float *nxt, float *cnxt, double &res, double &dang) {
    float nx;
    if (ps.personalized) {
        nx = __fmul_rn(ps.damping, sum);
        if (r == ps.source) nx = __fadd_rn(ps.tele, nx);
    } else {
        nx = __fadd_rn(ps.dshare, __fmul_rn(ps.damping, sum));
    }
    const float old = cur[r];
    res += fabs(static_cast<double>(nx) - static_cast<double>(old));
    nxt[r] = nx;
    const uint32_t od = a.out_deg[r];
    cnxt[r] = od ? __fdiv_rn(nx, static_cast<float>(od)) : 0.0f;
    if (od == 0) dang += static_cast<double>(nx);
}

// In-edge batches per lane of one gather pass of long and wide rows.
#ifndef HYT_PR_BATCH
#define HYT_PR_BATCH 8
#endif
constexpr int kBatch = HYT_PR_BATCH;

// Where a task reads its contributions: whole-vector array for untagged
// sources (L2, evict-last), table of the hot sources for tagged ones.  Slot
// num_hot of the table is 0: `none`, its tagged id, stands for "no edge".
// kSmemHot: the table is in shared memory; else in global memory, at most 2^31
// elements behind the array, and `turn` makes a tagged id an index of it from there.
struct Sources {
    const float *ccur;
    const float *hot;
    uint32_t none, turn;
    uint64_t pol;
};

__device__ __forceinline__ Sources make_sources(const PRArgs &a, const float *ccur, const float *hot) {
    return Sources{ccur, hot, kHotTag | a.num_hot, static_cast<uint32_t>(hot - ccur) - kHotTag, dev::policy_evict_last()};
}

// Loads one source's contribution: its bits end in `g | id`.  Not through the
// read-only path: the persistent solver rewrites the vector between
// iterations.  With the table in shared memory the two loads are predicated on
// the tag and write registers of their own (the hot one its id's), so that
// neither waits for the other and no branch splits a run of gathers; in global
// memory one load serves both.
template <bool kSmemHot>
__device__ __forceinline__ void load_contribution(uint32_t &id, uint32_t &g, const Sources &S) {
    g = 0;
    if constexpr (kSmemHot) {
        const uint32_t at = static_cast<uint32_t>(__cvta_generic_to_shared(S.hot)) + (id << 2);  // drops the tag
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %1, 0;\n\t"
            "@!p ld.global.L2::cache_hint.b32 %0, [%2], %3;\n\t"
            "@!p mov.b32 %1, 0;\n\t"
            "@p ld.shared.b32 %1, [%4];\n\t}"
            : "+r"(g), "+r"(id)
            : "l"(S.ccur + id), "l"(S.pol), "r"(at));
    } else {
        const uint32_t at = (id & kHotTag) ? id + S.turn : id;
        asm volatile("ld.global.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(g) : "l"(S.ccur + at), "l"(S.pol));
        id = 0;
    }
}

// Adds the kK contributions loaded by load_contribution.
template <int kK>
__device__ __forceinline__ void add_contributions(const uint32_t (&id)[kK], const uint32_t (&g)[kK], dev::CSum2 &acc) {
#pragma unroll
    for (int k = 0; k < kK; k += 2) acc.add(__uint_as_float(g[k] | id[k]), __uint_as_float(g[k + 1] | id[k + 1]));
}

// Adds the contributions of edges src[base + 32k + lane], k < kK, below n
// (kFull: all of them are).  Each of the kK id loads is one coalesced
// 128-byte access, and because the sources of an in-row are sorted, the 32
// addresses of each gather instruction are ascending and neighbouring lanes
// often share an L2 sector (dense for hub-heavy rows).  All kK gathers of a
// lane are issued before any is consumed.
template <int kK, bool kSmemHot, bool kFull>
__device__ __forceinline__ void gather_pass(const uint32_t *src, uint32_t base, uint32_t n, const Sources &S, int lane,
                                            dev::CSum2 &acc) {
    uint32_t id[kK];
#pragma unroll
    for (int k = 0; k < kK; ++k) {
        const uint32_t i = base + 32 * k + lane;
        id[k] = (kFull || i < n) ? dev::ld_stream(src + i) : S.none;
    }
    uint32_t g[kK];
#pragma unroll
    for (int k = 0; k < kK; ++k) load_contribution<kSmemHot>(id[k], g[k], S);
    add_contributions<kK>(id, g, acc);
}

// Adds the contributions of edges [0, n) of src.  The last, partial pass
// issues only the 4-batch groups that hold edges (a warp-uniform choice).
template <bool kSmemHot>
__device__ __forceinline__ void gather_span(const uint32_t *src, uint32_t n, const Sources &S, int lane,
                                            dev::CSum2 &acc) {
    static_assert(kBatch % 4 == 0 && kBatch >= 4, "batches come in groups of 4");
    uint32_t base = 0;
    for (; base + 32 * kBatch <= n; base += 32 * kBatch) gather_pass<kBatch, kSmemHot, true>(src, base, n, S, lane, acc);
    if (base == n) return;
    const uint32_t groups = (n - base + 127) / 128;  // 4-batch groups holding edges
    if (groups == 1)
        gather_pass<4, kSmemHot, false>(src, base, n, S, lane, acc);
    else if (groups == 2)
        gather_pass<8, kSmemHot, false>(src, base, n, S, lane, acc);
    else
        gather_pass<kBatch, kSmemHot, false>(src, base, n, S, lane, acc);
}

// Stop rule of iteration `it` (thread 0 of the last CTA, or the separate
// end kernel): residual <= tolerance or the iteration cap.
__device__ __forceinline__ void end_iteration(const PRArgs &a, uint32_t it) {
    const double r = atomicAdd(&a.residual[it], 0.0);
    const uint32_t n_it = it + 1;
    const bool conv = r <= static_cast<double>(a.tolerance);
    a.hdr->last_residual = r;
    a.hdr->iter = n_it;
    if (conv || n_it >= a.max_iter) {
        a.hdr->done = 1;
        a.hdr->converged = conv ? 1u : 0u;
    }
}


// Ends iteration `it` on the device (any thread): the stop rule with the
// iteration's reduced residual.
__device__ __forceinline__ void close_iteration(const PRArgs &a, uint32_t it, double residual, double dangling) {
    a.residual[it] = residual;
    a.dangling[it + 1] = dangling;
    const uint32_t n_it = it + 1;
    const bool conv = residual <= static_cast<double>(a.tolerance);
    a.hdr->last_residual = residual;
    a.hdr->iter = n_it;
    if (conv || n_it >= a.max_iter) {
        a.hdr->done = 1;
        a.hdr->converged = conv ? 1u : 0u;
    }
}

// Records task slot `slot`'s (res, dang); lane 0 stores, no wait.
__device__ __forceinline__ void slot_store(double2 *slots, uint32_t slot, double res, double dang, int lane) {
    if (lane == 0) slots[slot] = make_double2(res, dang);
}

// Solver scalars of an iteration whose dangling mass (sum of x over
// out-degree-0 vertices) is dmass.
__device__ __forceinline__ PRState make_state(const PRArgs &a, double dmass) {
    PRState ps;
    ps.damping = a.damping;
    ps.source = a.source;
    ps.personalized = a.personalized != 0;
    ps.dshare = __fadd_rn(a.base, static_cast<float>(static_cast<double>(a.damping) * dmass / static_cast<double>(a.V)));
    ps.tele = static_cast<float>((1.0 - static_cast<double>(a.damping)) + static_cast<double>(a.damping) * dmass);
    return ps;
}

// Rank buffers of iteration `it` (Jacobi double buffering by parity).
struct PRBuffers {
    const float *cur, *ccur;
    float *nxt, *cnxt;
};

__device__ __forceinline__ PRBuffers buffers(const PRArgs &a, uint32_t it) {
    PRBuffers b;
    b.cur = (it & 1) ? a.rank[1] : a.rank[0];
    b.nxt = (it & 1) ? a.rank[0] : a.rank[1];
    b.ccur = (it & 1) ? a.contrib[1] : a.contrib[0];
    b.cnxt = (it & 1) ? a.contrib[0] : a.contrib[1];
    return b;
}

// What a pull task works on: edges [e0, e0 + n); a tile's rows [a, b), or a
// chunk's long-row index a and chunk number b.
struct TaskSpan {
    uint64_t e0;
    uint32_t n, a, b;
};

__device__ __forceinline__ TaskSpan task_span(uint4 d) {
    return TaskSpan{task_first_edge(d), task_edges(d), d.z, d.w};
}

// The same from the graph's tables, for callers that hold no descriptor.
__device__ __forceinline__ TaskSpan chunk_span(const PRArgs &a, uint64_t ci) {
    const uint2 t = a.chunk_tasks[ci];
    const uint32_t row = a.long_rows[t.x].row;
    const uint64_t lo = a.in_off[row] + uint64_t(t.y) * a.chunk_edges, re = a.in_off[row + 1];
    return TaskSpan{lo, static_cast<uint32_t>((lo + a.chunk_edges < re ? lo + a.chunk_edges : re) - lo), t.x, t.y};
}

__device__ __forceinline__ TaskSpan tile_span(const PRArgs &a, uint64_t k) {
    const uint32_t r0 = a.tile_start[k], r1 = a.tile_start[k + 1];
    if (r0 == r1) return TaskSpan{0, 0, r0, r0};
    const uint64_t last_b = a.in_off[r1 - 1], last_e = a.in_off[r1];
    const bool chunked = last_e - last_b >= a.tile_cost;  // a long last row is chunked
    const uint64_t e0 = a.in_off[r0];
    return TaskSpan{e0, static_cast<uint32_t>((chunked ? last_b : last_e) - e0), r0, chunked ? r1 - 1 : r1};
}

// Chunk task: a chunk_edges-edge slice of a long row.  The warp stores its
// compensated partial; the last arriving warp of the row merges every partial
// in chunk order (lane j takes chunks j, j+32, ...) and finalizes the row.
// Returns the row's long-row index when this warp finalized it (lane 0 holds
// res/dang), else ~0u.  Must be called by all 32 lanes.
template <bool kSmemHot>
__device__ __forceinline__ uint32_t chunk_task(const PRArgs &a, const PRState &ps, const PRBuffers &b,
                                               const uint32_t *in_src, const float *s_hot, const TaskSpan &t, int lane,
                                               double &res, double &dang, const uint4 *prefetch = nullptr) {
    dev::CSum2 acc2;
    const LongRow L = a.long_rows[t.a];
    if (prefetch) prefetch_task(*prefetch, in_src, nullptr, lane);
    gather_span<kSmemHot>(in_src + t.e0, t.n, make_sources(a, b.ccur, s_hot), lane, acc2);
    const dev::CSum acc = dev::warp_reduce(acc2.total());
    if (L.num_chunks == 1) {  // the whole row: nothing to merge
        if (lane == 0) finalize_row(a, ps, L.row, acc.value(), b.cur, b.nxt, b.cnxt, res, dang);
        return t.a;
    }
    uint32_t last = 0;
    if (lane == 0) {
        a.partial[L.first_chunk + t.b] = make_float2(acc.s, acc.c);
        __threadfence();
        const uint32_t tk = atomicAdd(&a.ticket[t.a], 1u) + 1u;
        last = (tk % L.num_chunks == 0) ? 1u : 0u;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return ~0u;
    __threadfence();
    dev::CSum row;
    for (uint32_t j = lane; j < L.num_chunks; j += 32) {
        const float2 p = __ldcg(a.partial + L.first_chunk + j);
        dev::CSum x;
        x.s = p.x;
        x.c = p.y;
        row.merge(x);
    }
    row = dev::warp_reduce(row);
    if (lane == 0) finalize_row(a, ps, L.row, row.value(), b.cur, b.nxt, b.cnxt, res, dang);
    return t.a;
}

// One group step of a tile's short rows: kG lanes per row, 32 / kG rows at a
// time (the step's rows belong to lanes step * 32 / kG ... of the batch).
// Lane l of a row takes edges lo + l, lo + l + kG, ..., up to kEdges of them,
// all in flight (rows have at most kG * kEdges in-edges here); the group's compensated sums merge by shuffles.  Returns the
// row's sum to the lane that owns it (other lanes keep `sum`).
template <int kG, int kEdges, bool kSmemHot>
__device__ __forceinline__ float group_step(const uint32_t *src, uint32_t lo, uint32_t hi, int step, const Sources &S,
                                            int lane, float sum) {
    constexpr int kRows = 32 / kG;   // rows of one step
    const int owner = step * kRows + lane / kG;
    const uint32_t b = __shfl_sync(0xffffffffu, lo, owner) + (lane % kG);
    const uint32_t e = __shfl_sync(0xffffffffu, hi, owner);
    uint32_t id[kEdges];
#pragma unroll
    for (int j = 0; j < kEdges; ++j) id[j] = (b + j * kG < e) ? dev::ld_stream(src + b + j * kG) : S.none;
    uint32_t g[kEdges];
#pragma unroll
    for (int j = 0; j < kEdges; ++j) load_contribution<kSmemHot>(id[j], g[j], S);
    dev::CSum2 acc2;
    add_contributions<kEdges>(id, g, acc2);
    dev::CSum acc = acc2.total();
#pragma unroll
    for (int o = 1; o < kG; o <<= 1) {
        dev::CSum w;
        w.s = __shfl_xor_sync(0xffffffffu, acc.s, o);
        w.c = __shfl_xor_sync(0xffffffffu, acc.c, o);
        acc.merge(w);
    }
    const float t = __shfl_sync(0xffffffffu, acc.value(), (lane % kRows) * kG);
    return lane / kRows == step ? t : sum;
}

template <int kG, int kEdges, bool kSmemHot>
__device__ __forceinline__ float group_rows(const uint32_t *src, uint32_t lo, uint32_t hi, const Sources &S, int lane) {
    float sum = 0.0f;
    for (int step = 0; step < kG; ++step) sum = group_step<kG, kEdges, kSmemHot>(src, lo, hi, step, S, lane, sum);
    return sum;
}

// Tile task: rows [t.a, t.b), 32 at a time, one per lane: bounds, rank and
// out-degree are loaded coalesced (the next batch's before this one's
// gathers), in-edge sums are taken from registers, and every lane finalizes
// its row.  Rows of kWarpRowDegree or more in-edges are summed by the whole
// warp one after another; the others by groups of 1, 2, 4 or 8 lanes, the
// smallest that leaves each lane at most 8 edges of the batch's largest row
// (one round of loads per row; larger groups leave lanes idle, and 16 lanes
// for rows of 64 to 127 ran 5 to 15 % slower than the warp on R-MAT scale
// 24).  Must be called by all 32 lanes.
// prefetch (optional): the warp's next pull task, whose edge lines are
// warmed in L2 (warming its rows' offsets and ranks too gained nothing).
// kPart: the task is a part of a tile, cut where out-of-HBM pieces are.  Its
// rows keep the batches, and so the lanes per row and the last bits, that they
// have in the whole tile, rows [whole.x, whole.y): a row's sum depends on the
// largest row beside it.
template <bool kSmemHot, bool kPart = false>
__device__ __forceinline__ void tile_task(const PRArgs &a, const PRState &ps, const PRBuffers &b,
                                          const uint32_t *in_src, const float *s_hot, const TaskSpan &t, int lane,
                                          double &res, double &dang, const uint4 *prefetch = nullptr,
                                          uint2 whole = make_uint2(0, 0)) {
    const uint32_t r0 = t.a, rl = t.b;
    if (r0 == rl) return;
    const uint64_t e0 = t.e0;
    const uint32_t *src = in_src + e0;
    const Sources S = make_sources(a, b.ccur, s_hot);
    uint32_t lo = 0, hi = 0, od = 0;  // this lane's row: bounds relative to e0, out-degree, rank
    uint32_t beside = 0;              // in-edges of a row of the tile's other parts
    float old = 0.0f;
    auto load_row = [&](uint32_t r, uint32_t &l, uint32_t &h, uint32_t &d, float &o, uint32_t &bs) {
        l = h = d = bs = 0;
        o = 0.0f;
        if ((!kPart || r >= r0) && r < rl) {
            l = static_cast<uint32_t>(a.in_off[r] - e0);
            h = static_cast<uint32_t>(a.in_off[r + 1] - e0);
            o = b.cur[r];
            d = a.out_deg[r];
        } else if (kPart && r < whole.y) {
            bs = static_cast<uint32_t>(a.in_off[r + 1] - a.in_off[r]);
        }
    };
    const uint32_t rfirst = kPart ? whole.x + ((r0 - whole.x) & ~31u) : r0;
    load_row(rfirst + lane, lo, hi, od, old, beside);
    if (prefetch) prefetch_task(*prefetch, in_src, nullptr, lane);
    for (uint32_t rb = rfirst; rb < rl; rb += 32) {
        uint32_t lo_n, hi_n, od_n, beside_n;
        float old_n;
        load_row(rb + 32 + lane, lo_n, hi_n, od_n, old_n, beside_n);
        const uint32_t deg = kPart ? hi - lo + beside : hi - lo;
        const bool wide = deg >= kWarpRowDegree;
        const uint32_t most = __reduce_max_sync(0xffffffffu, wide ? 0u : deg);
        const uint32_t hs = wide ? lo : hi;  // group steps see a wide row as empty
        float sum = 0.0f;
        if (most > 32)
            sum = group_rows<8, 8, kSmemHot>(src, lo, hs, S, lane);
        else if (most > 16)
            sum = group_rows<4, 8, kSmemHot>(src, lo, hs, S, lane);
        else if (most > 8)
            sum = group_rows<2, 8, kSmemHot>(src, lo, hs, S, lane);
        else if (most > 4)
            sum = group_rows<1, 8, kSmemHot>(src, lo, hs, S, lane);
        else if (most > 2)
            sum = group_rows<1, 4, kSmemHot>(src, lo, hs, S, lane);
        else if (most)
            sum = group_rows<1, 2, kSmemHot>(src, lo, hs, S, lane);
        uint32_t big = __ballot_sync(0xffffffffu, wide && (!kPart || !beside));
        while (big) {
            const int w = __ffs(big) - 1;
            big &= big - 1;
            const uint32_t bb = __shfl_sync(0xffffffffu, lo, w);
            const uint32_t ee = __shfl_sync(0xffffffffu, hi, w);
            dev::CSum2 acc;
            gather_span<kSmemHot>(src + bb, ee - bb, S, lane, acc);
            const float t = dev::warp_reduce(acc.total()).value();
            if (lane == w) sum = t;
        }
        if ((!kPart || rb + lane >= r0) && rb + lane < rl) finalize_row_with(ps, rb + lane, sum, old, od, b.nxt, b.cnxt, res, dang);
        lo = lo_n;
        hi = hi_n;
        od = od_n;
        old = old_n;
        beside = beside_n;
    }
}

}  // namespace prc
}  // namespace hyt
