// Single-source shortest paths: frontier push over the CSR with atomicMin.
//
// The reference solver (src/algorithms/sssp.cpp:109-234, cuda/sssp.cu:
// 100-154) is a synchronous Bellman-Ford that pulls over all in-edges every
// round.  Any label-correcting schedule reaches the same fixed point
//     d[s] = 0,  d[v] = min_{u->v} (d[u] + w(u,v))
// because every relaxation only lowers a label to a value that some path
// attains; so distances are bit-identical to the reference.  Integer (u32)
// weights relax with exact integer adds; float weights relax with the same
// IEEE add the reference uses, compared as ordered bit patterns (valid for
// non-negative floats).
//
// Schedule: near/far buckets (Delta-stepping with one far pile).  Vertices
// whose label drops below the current threshold T join the next near
// frontier; the others go to the far pile.  When the near frontier runs
// dry, T grows by Delta and the far pile is split: entries now below T
// become the near frontier, entries below the old threshold are stale
// (already settled) and are dropped.  Delta = infinity is plain frontier
// Bellman-Ford (used for float weights).
//
// Expansion is warp-centric: a warp takes 32 frontier vertices, prefix-sums
// their degrees with shuffles and walks the combined edge list 32 edges at
// a time, finding each edge's owner with a 5-step shuffle binary search.
// Rows of >= kHubDegree edges become kHubChunk-edge warp tasks for a second
// grid-wide kernel, so no warp owns more than ~2K edges of a round.  Each
// lane keeps 8 or 16 edges in flight through loads and atomics (relax_batch).  A
// vertex joins a frontier once per round (round stamp) and the far pile once
// per phase (phase stamp), appended with one warp-aggregated atomic.
//
// With one bucket and a CSC, a round whose frontier carries more than
// E / pull_div out-edges runs as a pull sweep over the CSC instead
// (sssp_pull_kernel: rows take their minimum from registers, sssp_pull.cuh;
// tile rows are written with plain stores).  Staging a tile's candidates in
// 132 KB of shared memory left the label gathers too little L1 for their
// outstanding misses; without it, and with the next frontier's out-edges and
// lowest label summed by the kernels that fill it, a solve of R-MAT scale 24
// went from 4.76 to 4.33 ms.  A sweep skips the rows whose label
// is at most (lowest frontier label + smallest weight): no in-edge can
// lower them, so their in-edges are neither read nor gathered.  All round
// state lives on the device; with one bucket the whole solve is one
// cooperative launch (sssp_solve_kernel), with a finite bucket width the
// rounds run as a conditional CUDA graph (split, expand, hub chunks, round
// end), instantiated once per graph and launched again by later solves.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>
#include <utility>

#include "common.cuh"
#include "graph.cuh"
#include "grid_sync.cuh"
#include "host_checks.hpp"
#include "scratch.cuh"
#include "hybrid.cuh"
#include "solvers.cuh"
#include "sssp_core.cuh"
#include "sssp_pull.cuh"

namespace hyt {
namespace {

using namespace ssc;

// Splits the far pile at the start of a round whose near frontier is empty.
__global__ void __launch_bounds__(kSSThreads) sssp_split_kernel(const SSArgs *__restrict__ args) {
    const SSArgs a = *args;
    const SSHeader *h = a.hdr;
    if (*(volatile const uint32_t *)&h->done || !*(volatile const uint32_t *)&h->pending) return;
    const uint32_t n = (h->phase & 1) ? h->fsize[1] : h->fsize[0];
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) split_entry(a, i);
}

// HYB: the edges of a vertex's partition are reached through a.loc
// (partitioned solves); compacted partitions are expanded from their packed
// payload by sssp_expand_packed_kernel instead.
// TRACK: pull-capable solves (the kernel also gathers the next frontier's
// out-edges and lowest label).
template <int WK, bool HYB = false, bool TRACK = false>
__global__ void __launch_bounds__(kSSThreads) sssp_expand_kernel(const SSArgs *__restrict__ args) {
    const SSArgs a = *args;
    if (*(volatile uint32_t *)&a.hdr->done || pull_round(a)) return;
    const RoundView rv = round_view(a);
    const int lane = threadIdx.x & 31;
    const uint32_t gwarp = (blockIdx.x * kSSThreads + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * kSSThreads) >> 5;
    unsigned long long relaxed = 0, improved = 0;
    auto hub = [&](uint32_t v, uint32_t nch) {
        const uint32_t base = atomicAdd(&a.hdr->hub_count, nch);
        for (uint32_t c = 0; c < nch; ++c) a.hubs[base + c] = make_uint2(v, c);
    };
    Gain gain;
    for (uint32_t w = gwarp; uint64_t(w) * 32 < rv.qn; w += nwarps)
        expand_warp<WK, HYB, HYB ? kEdgeBatch : 16, TRACK>(a, rv, w * 32, lane, kHubDegree, relaxed, improved, hub,
                                                           &gain);
    if constexpr (TRACK) flush_gain(a, gain, lane);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) relaxed += __shfl_xor_sync(0xffffffffu, relaxed, o);
    if (lane == 0 && relaxed) atomicAdd(&a.hdr->relaxations, relaxed);
}

// One warp per kHubChunk-edge slice of a long frontier row.
template <int WK, bool HYB = false, bool TRACK = false>
__global__ void __launch_bounds__(kSSThreads) sssp_hub_kernel(const SSArgs *__restrict__ args) {
    const SSArgs a = *args;
    if (*(volatile uint32_t *)&a.hdr->done || pull_round(a)) return;
    const RoundView rv = round_view(a);
    const uint32_t n = *(volatile uint32_t *)&a.hdr->hub_count;
    const int lane = threadIdx.x & 31;
    const uint32_t gwarp = (blockIdx.x * kSSThreads + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * kSSThreads) >> 5;
    unsigned long long improved = 0;
    Gain gain;
    for (uint32_t t = gwarp; t < n; t += nwarps) {
        const uint2 h = a.hubs[t];
        const uint32_t *hc = a.cols, *hw = a.weights;
        if constexpr (HYB) {
            const EdgeLoc L = a.loc[h.x >> a.part_shift];
            hc = L.cols;
            hw = L.weights;
        }
        hub_chunk<WK, TRACK>(a, rv, hc, hw, h.x, h.y, lane, improved, &gain);
    }
    if constexpr (TRACK) flush_gain(a, gain, lane);
}

// ---- pull sweeps (direction-optimised rounds) ------------------------------
//
// A round whose frontier carries more than E / pull_div out-edges is run as
// a sweep over the CSC instead: every vertex takes the minimum of
// d[u] + w(u, v) over its in-edges (no atomics on the edge path, streaming
// reads of ids and weights, label gathers from L2), and improved vertices
// form the next frontier.  Any label-correcting schedule reaches the same
// fixed point, so distances are unchanged.  Single-bucket solves only.

// CSC of the graph for pull sweeps (PageRank's tiles and long-row chunks).
struct PullGraph {
    const uint64_t *in_off;
    const uint32_t *in_src;   // hot sources tagged kHotTag | slot
    const uint32_t *in_w;     // weights in CSC order (NULL when unweighted), or packed words
    const LongRow *long_rows;
    const uint32_t *hot_vertex;
    const uint4 *tasks;       // pull task descriptors: chunks of long rows, then tiles
    uint64_t num_tasks;
    uint64_t dealt;           // tasks dealt to the warps in turn; the rest go to whoever is free
    uint32_t num_hot;
    uint32_t bits;            // packed words: bits of the source id
};


// Lowers tile row r's label from `seen` to c if that improves it; true when
// r joins the next frontier.  A tile row has exactly one writer during a
// sweep (the warp that owns its tile) and no push runs beside a sweep, so
// `seen` -- read before the tile's gathers -- is the row's label, and plain
// stores replace the atomics.
__device__ __forceinline__ bool pull_store(const SSArgs &a, const RoundView &rv, uint32_t r, uint32_t c,
                                           uint32_t seen) {
    if (c >= seen) return false;
    a.dist[r] = c;
    a.stamp[r] = rv.next_stamp;
    return true;
}

// Lowers row r's label to c; true when that improved it, `joined` when r
// joins the next frontier for the first time this round.
__device__ __forceinline__ bool pull_relax(const SSArgs &a, const RoundView &rv, uint32_t r, uint32_t c, bool &joined) {
    if (c >= __ldcg(a.dist + r) || c >= atomicMin(a.dist + r, c)) return false;
    joined = atomicExch(a.stamp + r, rv.next_stamp) != rv.next_stamp;
    return true;
}

// One CTA per SM.  768 threads leave 80 registers: 1024 spill in the whole-solve
// kernel and make every grid barrier wait for more warps.  Threads 1024 / 896 /
// 768 / 640 / 512, one source: R-MAT 16 M vertices 2.34 / 2.35 / 2.34 / 2.42 /
// 2.65 ms, 1 M 565 / 549 / 511 / 504 / 552 us, 2 M in input order 675 / 650 /
// 650 / 688 / 714 us, 4099 vertices 323 / 322 / 300 / 272 / 267 us (one box
// each side of 768).  Loading a step's ids ahead, as the multi-source sweep
// does, was slower at every size (2.41 ms and up at 16 M).
constexpr int kPullThreads = 768;
// A whole solve with fewer tasks than the GPU has warps runs with smaller CTAs, down
// to 16 warps: its rounds are barriers, which wait for every warp, while fewer
// warps mean more CTAs to meet.  At least 24 / 16 / 8 / 4 warps: 4099 vertices in
// input order 312 / 300 / 298 / 325 us, in hub order 241 / 239 / 261 / 288 us,
// 16001 in hub order 225 / 215 / 212 / 220 us; from 131 K vertices on all are the
// same.
constexpr uint64_t kMinWarps = 16;

// Row skipping.  Let F be this round's frontier (every vertex whose label
// dropped since its out-edges were last relaxed) and fmin its lowest label.
// An in-edge (u, v) can lower d[v] this round only if u is in F, and then
// its candidate is d[u] + w >= fmin + min_w.  So a row with
// d[v] <= extend(fmin, min_w) cannot improve: its in-edges are neither
// read nor gathered.  A vertex lowered during the round joins the next
// frontier, so the argument holds again next round; distances are
// unchanged.
template <int WK>
__device__ __forceinline__ uint32_t skip_bound(const SSArgs &a, uint32_t fmin, bool &on) {
    on = a.skip_rows && fmin < a.inf;
    return on ? extend<WK>(fmin, a.min_w) : 0u;
}

// One sweep over the whole grid.  fmin: the frontier's lowest label; relaxed
// and gain are added to (chunks counted by lane 0, tile rows by their lanes).
// Labels are read live, not from a snapshot: rows lowered early in a sweep
// feed the rows after them (a snapshot of the hottest labels in shared memory
// cost a round).
// Tasks cost uneven amounts (rows skipped, mixed degrees), so only the first
// pg.dealt are dealt in turn; the others are taken one by one from `cursor`
// (on R-MAT in input order a quarter of the warps' time went idle at the end
// of a sweep).
template <int WK, bool kPacked>
__device__ __forceinline__ void pull_sweep(const SSArgs &a, const PullGraph &pg, const RoundView &rv, uint32_t fmin,
                                           const uint32_t *s_hot, uint32_t *cursor, unsigned long long &relaxed,
                                           Gain &gain) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t pol = dev::policy_evict_last();
    const auto label = [&](uint32_t u) { return dev::ld_keep_u32(a.dist + u, pol); };
    const uint64_t nwarps = uint64_t(gridDim.x) * (blockDim.x / 32);
    const uint32_t *pf_a = kPacked ? pg.in_w : pg.in_src;
    const uint32_t *pf_w = (kPacked || WK == HYT_WEIGHTS_NONE) ? nullptr : pg.in_w;
    bool skip_on;
    const uint32_t skip_at = skip_bound<WK>(a, fmin, skip_on);
    const uint64_t dealt = max(pg.dealt, min(pg.num_tasks, nwarps));  // every warp's first task is dealt
    uint64_t task = uint64_t(blockIdx.x) * (blockDim.x / 32) + warp;
    // each dealt task's descriptor is read while the task before it runs
    uint4 d = task < pg.num_tasks ? pg.tasks[task] : make_uint4(0, 0, 0, 0);
    while (task < pg.num_tasks) {
        // the next task: dealt, or asked for now and looked at when this one is done
        uint64_t next = task + nwarps;
        uint32_t ticket = 0;
        const bool ask = next >= dealt;
        if (ask && lane == 0) ticket = atomicAdd(cursor, 1u);
        uint4 nd = ask ? make_uint4(0, 0, 0, 0) : pg.tasks[next];
        const uint64_t e0 = task_first_edge(d);
        const ssp::InEdges E{pg.in_src + e0, (WK == HYT_WEIGHTS_NONE) ? nullptr : pg.in_w + e0, s_hot, pg.bits, a.inf};
        if (task_is_chunk(d)) {
            // slice of a long row: warp minimum, then one relaxation
            const uint32_t r = pg.long_rows[d.z].row, n = task_edges(d);
            if (!ask) prefetch_task(nd, pf_a, pf_w, lane);
            if (!(skip_on && __shfl_sync(0xffffffffu, __ldcg(a.dist + r), 0) <= skip_at)) {
                const uint32_t best = ssp::span_min<WK, kPacked>(E, 0, n, label, lane);
                if (lane == 0) {
                    relaxed += n;
                    if (best < a.inf) {
                        bool joined = false;
                        if (pull_relax(a, rv, r, best, joined)) gain.low = min(gain.low, best);
                        if (joined) {
                            gain.edges += a.out_deg[r];
                            append(rv.qnext, rv.qnext_size, r);
                        }
                    }
                }
            }
        } else {
            // merge-path tile of short rows, 32 at a time, one per lane: the
            // next batch's bounds and labels load before this one's gathers
            const uint32_t rl = d.w;
            uint32_t lo = 0, hi = 0, seen = 0;
            auto load_row = [&](uint32_t r, uint32_t &l, uint32_t &h, uint32_t &sn) {
                l = h = sn = 0;
                if (r < rl) {
                    l = static_cast<uint32_t>(pg.in_off[r] - e0);
                    h = static_cast<uint32_t>(pg.in_off[r + 1] - e0);
                    sn = __ldcg(a.dist + r);
                }
            };
            load_row(d.z + lane, lo, hi, seen);
            if (!ask) prefetch_task(nd, pf_a, pf_w, lane);
            for (uint32_t rb = d.z; rb < rl; rb += 32) {
                uint32_t lo_n, hi_n, seen_n;
                load_row(rb + 32 + lane, lo_n, hi_n, seen_n);
                const uint32_t r = rb + lane;
                if (skip_on && seen <= skip_at) hi = lo;  // no in-edge can lower it: neither read nor gathered
                relaxed += hi - lo;
                const uint32_t best = ssp::rows_min<WK, kPacked>(E, lo, hi, label, lane);
                const bool joined = r < rl && pull_store(a, rv, r, best, seen);
                if (joined) {
                    gain.low = min(gain.low, best);
                    gain.edges += a.out_deg[r];
                }
                const uint32_t vals[1] = {r};
                warp_append<1>(rv.qnext, rv.qnext_size, vals, joined ? 1u : 0u, lane);
                lo = lo_n;
                hi = hi_n;
                seen = seen_n;
            }
        }
        if (ask) {
            next = dealt + __shfl_sync(0xffffffffu, ticket, 0);
            if (next < pg.num_tasks) nd = pg.tasks[next];
        }
        task = next;
        d = nd;
    }
}

// Vertex ids of the hot slots into shared memory.
__device__ __forceinline__ void load_hot_ids(const PullGraph &pg, uint32_t *s_hot) {
    for (uint32_t i = threadIdx.x; i < pg.num_hot; i += blockDim.x) s_hot[i] = pg.hot_vertex[i];
    __syncthreads();
}

__device__ __forceinline__ void flush_relaxed(const SSArgs &a, unsigned long long relaxed, int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) relaxed += __shfl_xor_sync(0xffffffffu, relaxed, o);
    if (lane == 0 && relaxed) atomicAdd(&a.hdr->relaxations, relaxed);
}

// A sweep as a launch of its own (profiling and launch-by-launch runs).  a:
// the solve's arguments as kernel parameters (the constant bank: no registers
// held across the tasks).
template <int WK, bool kPacked>
__global__ void __launch_bounds__(kPullThreads, 1) sssp_pull_kernel(const __grid_constant__ SSArgs a,
                                                                    const __grid_constant__ PullGraph pg) {
    extern __shared__ __align__(16) uint32_t s_hot[];  // vertex ids of the hot slots (tagged sources in the CSC)
    if (*(volatile uint32_t *)&a.hdr->done || !pull_round(a)) return;
    load_hot_ids(pg, s_hot);
    unsigned long long relaxed = 0;
    Gain gain;
    pull_sweep<WK, kPacked>(a, pg, round_view(a), *(volatile const uint32_t *)&a.hdr->fmin, s_hot,
                            &a.hdr->task_cursor, relaxed, gain);
    flush_gain(a, gain, threadIdx.x & 31);
    flush_relaxed(a, relaxed, threadIdx.x & 31);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.hdr->pull_rounds, 1u);
}

// ---- a whole solve in one cooperative launch -------------------------------

// Totals of one round's frontier.  Three of them take turns: round r reads
// its own, fills the next round's and clears the one after (which every CTA
// left behind at the last barrier).
struct FrontierTotals {
    uint32_t qsize, hub_count, fmin_inv, task_cursor;
    unsigned long long edges;
};
struct SolveState {
    FrontierTotals round[3];
    uint32_t barrier, pad;
};

// 32-edge batches in flight of a push round's warp beside sweeps: 4 lose 5 % on
// 2^24 vertices, 16 spill and lose 10 %.
constexpr int kSolveBatch = 8;
// Solves that only push (no CSC, or no sweeps wanted) do without the sweep's code
// and the next frontier's out-degrees, a random read per improved vertex.  From
// kWideFrontierEdges on their frontiers are large enough for 16 batches a warp.
// Threads x batches 512 x 8 / 512 x 16 / 768 x 8 / the kernel with sweeps, one
// source: R-MAT 1 M vertices, 16 M edges 0.88 / 0.95 / 0.90 / 0.93 ms in input
// order, 0.99 / 1.10 / 1.01 / 1.05 in hub order; 16.7 M, 263 M 9.14 / 8.85 / 9.38 /
// 9.98 and 8.86 / 8.33 / 8.93 / 9.48; a grid of 1024 x 1024 11.1 / 13.9 / 12.6 /
// 15.1.
constexpr int kPushThreads = 512;
constexpr int kWideBatch = 16;
constexpr uint64_t kWideFrontierEdges = uint64_t(1) << 27;

// Rounds separated by grid barriers (one after a sweep; one between expansion
// and hub chunks and one after) in place of four launches and a conditional-
// graph step each, most of which found nothing to do: a solve of 65 K edges
// has 16 rounds (605 -> 318 us a call; 500 K vertices, 8 M edges: 935 -> 694
// us).  One bucket only; the loop of launches serves finite bucket
// widths.
// kPull: rounds may be sweeps.  kB: 32-edge batches in flight of a push round's warp.
template <int WK, bool kPacked, bool kPull, int kB>
__global__ void __launch_bounds__(kPull ? kPullThreads : kPushThreads, 1)
    sssp_solve_kernel(const __grid_constant__ SSArgs a, const __grid_constant__ PullGraph pg, SolveState *st,
                      uint32_t max_rounds) {
    extern __shared__ __align__(16) uint32_t s_hot[];
    const int lane = threadIdx.x & 31;
    const uint32_t gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    uint32_t barriers = 0;
    load_hot_ids(pg, s_hot);
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.V; v += gridDim.x * blockDim.x) {
        const bool s = v == a.source;
        a.dist[v] = s ? 0u : a.inf;
        a.stamp[v] = s ? 0u : 0xFFFFFFFFu;
    }
    if (lead) {
        a.queue[0][0] = a.source;
        st->round[0].qsize = 1;
        st->round[0].fmin_inv = ~0u;
        st->round[0].edges = a.row_off[a.source + 1] - a.row_off[a.source];
    }
    bool ok = dev::grid_sync(&st->barrier, barriers);
    unsigned long long relaxed = 0, frontier_total = 0;
    uint32_t sweeps = 0;
    for (uint32_t r = 0; ok; ++r) {
        FrontierTotals *cur = &st->round[r % 3], *nxt = &st->round[(r + 1) % 3];
        RoundView rv{};
        rv.r = r;
        rv.qn = __ldcg(&cur->qsize);
        if (rv.qn == 0 || r >= max_rounds) {
            if constexpr (kPacked)  // the solve's own infinity becomes the caller's
                for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.V; v += gridDim.x * blockDim.x)
                    if (__ldcg(a.dist + v) >= a.inf) a.dist[v] = HYT_DIST_INF_U32;
            if (lead) {
                a.hdr->round = r;
                a.hdr->converged = rv.qn == 0 ? 1u : 0u;
                a.hdr->frontier_total = frontier_total;
                a.hdr->pull_rounds = sweeps;
                a.hdr->done = 1;
            }
            flush_relaxed(a, relaxed, lane);
            return;
        }
        if (lead) st->round[(r + 2) % 3] = FrontierTotals{0, 0, 0, 0, 0};
        rv.threshold = 0xFFFFFFFFu;  // one bucket
        rv.next_stamp = r + 1;
        rv.q = a.queue[r & 1];
        rv.qnext = a.queue[(r + 1) & 1];
        rv.qnext_size = &nxt->qsize;
        rv.far = a.far[0];
        rv.far_size = &a.hdr->fsize[0];
        rv.far_stamp = 1;
        frontier_total += rv.qn;
        Gain gain;
        bool sweep = false;
        if constexpr (kPull) sweep = __ldcg(&cur->edges) * a.pull_div > a.num_edges;
        if (sweep) {
            if constexpr (kPull)
                pull_sweep<WK, kPacked>(a, pg, rv, ~__ldcg(&cur->fmin_inv), s_hot, &cur->task_cursor, relaxed, gain);
            ++sweeps;
        } else {
            unsigned long long improved = 0;
            auto hub = [&](uint32_t v, uint32_t nch) {
                const uint32_t base = atomicAdd(&cur->hub_count, nch);
                for (uint32_t c = 0; c < nch; ++c) a.hubs[base + c] = make_uint2(v, c);
            };
            for (uint32_t w = gwarp; uint64_t(w) * 32 < rv.qn; w += nwarps)
                expand_warp<WK, false, kB, kPull>(a, rv, w * 32, lane, kHubDegree, relaxed, improved, hub, &gain);
            ok = dev::grid_sync(&st->barrier, barriers);
            if (!ok) break;
            const uint32_t n = __ldcg(&cur->hub_count);
            for (uint32_t t = gwarp; t < n; t += nwarps) {
                const uint2 h = a.hubs[t];
                hub_chunk<WK, kPull, kB>(a, rv, a.cols, a.weights, h.x, h.y, lane, improved, &gain);
            }
        }
        if constexpr (kPull) flush_gain(&nxt->edges, &nxt->fmin_inv, gain, lane);
        ok = dev::grid_sync(&st->barrier, barriers);
    }
    if (threadIdx.x == 0) atomicExch(&a.hdr->error, 1u);
}

// End of a round of a pull-capable solve (one thread): the round's kernels
// have gathered the next frontier's out-edges (the next round's push / pull
// decision) and its lowest label while they filled it; a pass over the
// frontier for these took up to 0.1 ms a round on R-MAT scale 24.
__global__ void sssp_round_close_kernel(const SSArgs *__restrict__ args) {
    const SSArgs a = *args;
    SSHeader *h = a.hdr;
    if (h->done) return;
    const unsigned long long fe = h->frontier_edges_next;
    h->frontier_edges_next = 0;
    h->fmin = ~h->fmin_inv;  // all ones when the next frontier is empty
    h->fmin_inv = 0;
    h->task_cursor = 0;
    const bool finish = round_end(h);
    h->frontier_edges = fe;
    if (finish && a.use_cond) cudaGraphSetConditional(a.cond, 0);
}

// Unreached labels (inf or above) as the caller's infinity.
__global__ void sssp_unreached_kernel(uint32_t *dist, uint32_t V, uint32_t inf) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x)
        if (dist[v] >= inf) dist[v] = HYT_DIST_INF_U32;
}

__global__ void sssp_round_end_kernel(const SSArgs *__restrict__ args) {
    const SSArgs a = *args;
    if (a.hdr->done) return;
    if (round_end(a.hdr) && a.use_cond) cudaGraphSetConditional(a.cond, 0);
}

__global__ void sssp_init_kernel(const SSArgs *__restrict__ args) {
    const SSArgs a = *args;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < a.V; v += stride) init_vertex(a, v);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.queue[0][0] = a.source;
        a.hdr->frontier_edges = a.row_off[a.source + 1] - a.row_off[a.source];  // round 0's frontier
    }
}

// ---- partitioned (out-of-HBM) solves -------------------------------------

// Per-partition HyTM metrics of this round's frontier: active vertices,
// active edges (out-edges of active vertices), zero-copy requests
// ceil(deg * 4 / 128) and alignment overhead (row start not 128-byte aligned
// in the logical id array), as in the reference's cost model
// (src/transfer/hytm_cost_model.cpp:330-452).  Shared-memory histograms,
// one global atomic per CTA and partition.
constexpr uint32_t kMaxParts = 1024;

__global__ void __launch_bounds__(kSSThreads) sssp_part_stats_kernel(const SSArgs *__restrict__ args, uint32_t parts,
                                                                     PartMetrics *out) {
    __shared__ unsigned long long s_m[4 * kMaxParts];
    const SSArgs a = *args;
    for (uint32_t i = threadIdx.x; i < 4 * parts; i += blockDim.x) s_m[i] = 0;
    __syncthreads();
    const RoundView rv = round_view(a);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rv.qn; i += gridDim.x * blockDim.x) {
        const uint32_t v = rv.q[i];
        const uint32_t p = v >> a.part_shift;
        const uint64_t off = a.row_off[v];
        const uint64_t deg = a.row_off[v + 1] - off;
        atomicAdd(&s_m[4 * p + 0], 1ull);
        if (deg) {
            atomicAdd(&s_m[4 * p + 1], static_cast<unsigned long long>(deg));
            atomicAdd(&s_m[4 * p + 2], static_cast<unsigned long long>((deg * 4 + 127) / 128));
            if ((off * 4) % 128) atomicAdd(&s_m[4 * p + 3], 1ull);
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < 4 * parts; i += blockDim.x)
        if (s_m[i]) atomicAdd(reinterpret_cast<unsigned long long *>(out) + i, s_m[i]);
}

// Frontier vertices whose partition is compacted this round.
__global__ void sssp_compacted_list_kernel(const SSArgs *__restrict__ args, uint32_t *list, uint32_t *count) {
    const SSArgs a = *args;
    const RoundView rv = round_view(a);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rv.qn; i += gridDim.x * blockDim.x) {
        const uint32_t v = rv.q[i];
        if (a.loc[v >> a.part_shift].mode == kLocCompacted) append(list, count, v);
    }
}

// Expands the packed rows of compacted partitions (row i: vertex verts[i],
// edges [index[i], index[i+1]) of the packed cols / weights).
template <int WK>
__global__ void __launch_bounds__(kSSThreads) sssp_expand_packed_kernel(const SSArgs *__restrict__ args,
                                                                        CompactPayload pk) {
    const SSArgs a = *args;
    if (*(volatile uint32_t *)&a.hdr->done) return;
    const RoundView rv = round_view(a);
    const int lane = threadIdx.x & 31;
    const uint32_t gwarp = (blockIdx.x * kSSThreads + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * kSSThreads) >> 5;
    unsigned long long relaxed = 0, improved = 0;
    for (uint64_t w = gwarp; w * 32 < pk.rows; w += nwarps) {
        const uint64_t i = w * 32 + lane;
        uint32_t deg = 0, d = a.inf;
        uint64_t off = 0;
        if (i < pk.rows) {
            off = pk.index[i];
            deg = static_cast<uint32_t>(pk.index[i + 1] - off);
            d = __ldcg(a.dist + pk.verts[i]);
            relaxed += deg;
        }
        uint32_t incl = deg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        for (uint32_t base = 0; base < total; base += 32 * kEdgeBatch) {
            uint32_t u[kEdgeBatch], nd[kEdgeBatch], du[kEdgeBatch];
#pragma unroll
            for (int k = 0; k < kEdgeBatch; ++k) {
                const uint32_t j = base + 32 * k + lane;
                uint32_t lo = 0;
#pragma unroll
                for (uint32_t step = 16; step > 0; step >>= 1) {
                    const uint32_t probe = __shfl_sync(0xffffffffu, incl, lo + step - 1);
                    if (probe <= j) lo += step;
                }
                const uint32_t o_incl = __shfl_sync(0xffffffffu, incl, lo);
                const uint32_t o_deg = __shfl_sync(0xffffffffu, deg, lo);
                const uint64_t o_off = __shfl_sync(0xffffffffu, off, lo);
                const uint32_t o_d = __shfl_sync(0xffffffffu, d, lo);
                u[k] = 0;
                nd[k] = a.inf;
                if (j < total) {
                    const uint64_t e = o_off + (j - (o_incl - o_deg));
                    u[k] = dev::ld_stream(pk.cols + e);
                    nd[k] = extend<WK>(o_d, edge_weight<WK>(pk.weights, e));
                }
            }
#pragma unroll
            for (int k = 0; k < kEdgeBatch; ++k) du[k] = __ldcg(a.dist + u[k]);
            relax_batch<kEdgeBatch>(a, rv, u, nd, du, lane, improved);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) relaxed += __shfl_xor_sync(0xffffffffu, relaxed, o);
    if (lane == 0 && relaxed) atomicAdd(&a.hdr->relaxations, relaxed);
}

}  // namespace

// Row skipping in pull sweeps (env HYT_SSSP_PULL_SKIP, 0 = off; default on).
bool sssp_pull_skip() {
    static bool on = [] {
        const char *e = std::getenv("HYT_SSSP_PULL_SKIP");
        return !(e && e[0] == '0');
    }();
    return on;
}

namespace {

// Pull sweeps when the frontier's out-edges exceed E / div (env
// HYT_SSSP_PULL_DIV, 0 = never; default 4: a sweep reads every in-edge once,
// which costs about what pushing a quarter of them does).
uint32_t sssp_pull_div() {
    static uint32_t div = [] {
        const char *e = std::getenv("HYT_SSSP_PULL_DIV");
        return e ? static_cast<uint32_t>(std::strtoul(e, nullptr, 10)) : 4u;
    }();
    return div;
}

template <int WK, bool kPacked>
int pull_grid() {
    static int grid = 0;
    if (grid == 0) {
        int per_sm = 0;
        HYT_CUDA(cudaFuncSetAttribute(sssp_pull_kernel<WK, kPacked>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kPRSmemMax)));
        HYT_CUDA(cudaFuncSetAttribute(sssp_solve_kernel<WK, kPacked, true, kSolveBatch>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPRSmemMax)));
        HYT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sssp_pull_kernel<WK, kPacked>, kPullThreads,
                                                               kPRSmemMax));
        grid = sm_count() * std::max(per_sm, 1);
    }
    return grid;
}

template <int WK>
int expand_grid() {
    static int g = 0;
    if (g == 0) {
        int per_sm = 0;
        HYT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sssp_expand_kernel<WK>, kSSThreads, 0));
        g = sm_count() * std::max(per_sm, 1);
    }
    return g;
}

// kPacked: the graph keeps packed words, so its labels cannot wrap; sweeps use
// an infinity that leaves room for one more weight.
template <int WK, bool kPacked>
void sssp_solve(GraphImpl &g, uint32_t source, uint32_t delta, uint32_t max_rounds, uint32_t flags, cudaStream_t s,
                uint32_t *dist_out, hyt_run_stats *stats) {
    const uint64_t V = g.V;
    if (g.dist.count < V) g.dist.allocate(V);
    if (g.stamp.count < 2 * V) g.stamp.allocate(2 * V);
    for (int i = 0; i < 2; ++i) {
        if (g.queue[i].count < V) g.queue[i].allocate(V);
        if (g.far[i].count < V) g.far[i].allocate(V);
    }
    // each frontier vertex appears once per round: <= V rows, E/kHubChunk + V chunks
    const uint64_t hub_cap = V + g.E / kHubChunk + 2;
    if (g.hub_tasks.count < hub_cap) g.hub_tasks.allocate(hub_cap);
    static_assert(sizeof(SSArgs) <= 256 && sizeof(SSHeader) <= 256, "state block layout");
    const size_t sb = 512 + sizeof(SolveState);
    if (g.sssp_state.count < sb) g.sssp_state.allocate(sb);
    SSArgs *d_args = reinterpret_cast<SSArgs *>(g.sssp_state.get());
    SSHeader *hdr = reinterpret_cast<SSHeader *>(g.sssp_state.get() + 256);
    SolveState *solve_state = reinterpret_cast<SolveState *>(g.sssp_state.get() + 512);

    SSArgs a{};
    a.row_off = g.row_offsets.get();
    a.cols = g.cols.get();
    a.weights = g.weights.get();
    a.dist = g.dist.get();
    a.stamp = g.stamp.get();
    a.fstamp = g.stamp.get() + V;
    for (int i = 0; i < 2; ++i) {
        a.queue[i] = g.queue[i].get();
        a.far[i] = g.far[i].get();
    }
    a.hubs = g.hub_tasks.get();
    a.hdr = hdr;
    a.V = static_cast<uint32_t>(V);
    a.source = source;
    a.inf = (WK == HYT_WEIGHTS_F32) ? 0x7F800000u : HYT_DIST_INF_U32;
    a.num_edges = g.E;
    // pull sweeps need the CSC (and its weights) and a single bucket
    const bool pull_ok = (g.flags & HYT_GRAPH_PULL) && (WK == HYT_WEIGHTS_NONE || g.in_weights.get()) &&
                         delta == kNoDelta && g.E > 0;
    a.pull_div = pull_ok ? sssp_pull_div() : 0u;
    PullGraph pg{};
    if (a.pull_div) {
        pg.in_off = g.in_offsets.get();
        pg.in_src = g.in_sources.get();
        pg.in_w = g.in_weights.get();
        pg.long_rows = g.long_rows.get();
        pg.hot_vertex = g.hot_vertex.get();
        pg.tasks = g.pull_tasks.get();
        pg.num_tasks = g.num_chunks + g.num_tiles;
        pg.dealt = pg.num_tasks - pg.num_tasks / 4;  // skipped rows make tasks uneven in any vertex order
        pg.num_hot = kPacked ? 0u : g.num_hot;
        pg.bits = g.in_pack_bits;
        if (kPacked) a.inf = HYT_DIST_INF_U32 - g.weight_range.high;
    }
    a.out_deg = g.out_degree.get();
    // row skipping: the smallest edge weight bounds what any in-edge adds
    if (a.pull_div && sssp_pull_skip()) {
        a.skip_rows = 1;
        a.min_w = (WK == HYT_WEIGHTS_NONE) ? 1u : g.weight_range.low;
    }
    const unsigned pull_smem = static_cast<unsigned>(pg.num_hot * sizeof(uint32_t));
    const int pgrid = pull_grid<WK, kPacked>();

    SSHeader h0{};
    h0.qsize[0] = 1;
    h0.max_rounds = max_rounds;
    h0.delta = delta;
    h0.threshold = (WK == HYT_WEIGHTS_F32 || delta == kNoDelta) ? 0xFFFFFFFFu : delta;
    const bool far_pile = h0.threshold != 0xFFFFFFFFu;  // labels above the threshold wait in the far pile

    const bool in_graph = !(flags & HYT_RUN_NO_GRAPH) && !(flags & HYT_RUN_PROFILE);
    const bool persistent = in_graph && !far_pile;
    const int grid = expand_grid<WK>();
    // With a far pile the rounds are a conditional CUDA graph; an
    // instantiated loop of the same shape (kept with the graph object) is
    // launched again instead of being rebuilt.
    struct LoopKey {
        int wk, grid;
        const void *args;
    } key;
    std::memset(&key, 0, sizeof(key));
    key.wk = WK;
    key.grid = grid;
    key.args = d_args;
    LoopGraph &loop = g.sssp_loop;
    const bool reuse = in_graph && far_pile && loop.matches(&key, sizeof(key));
    if (in_graph && far_pile) {
        if (!reuse) {
            loop.reset();
            HYT_CUDA(cudaGraphCreate(&loop.graph, 0));
            HYT_CUDA(cudaGraphConditionalHandleCreate(&loop.cond, loop.graph, 1, cudaGraphCondAssignDefault));
        }
        a.cond = loop.cond;
        a.use_cond = 1;
    }

    EventTimer total;
    total.start(s);
    uint32_t launches = 1, hot = 0;
    double kernel_ms = 0.0;
    // split (finite bucket width), expand, hub, pull sweep + round close or round end
    const uint32_t per_round = (far_pile ? 1u : 0u) + 3u + (a.pull_div ? 1u : 0u);

    if (persistent) {
        HYT_CUDA(cudaMemsetAsync(hdr, 0, sizeof(SSHeader), s));
        HYT_CUDA(cudaMemsetAsync(solve_state, 0, sizeof(SolveState), s));
        // every CTA must be resident; no more of them than a sweep or a full
        // frontier has work for
        const uint64_t work = std::max<uint64_t>(pg.num_tasks, (V + 127) / 128);
        const void *solve = a.pull_div ? reinterpret_cast<void *>(sssp_solve_kernel<WK, kPacked, true, kSolveBatch>)
                            : g.E < kWideFrontierEdges
                                ? reinterpret_cast<void *>(sssp_solve_kernel<WK, false, false, kSolveBatch>)
                                : reinterpret_cast<void *>(sssp_solve_kernel<WK, false, false, kWideBatch>);
        const uint64_t warps = std::clamp<uint64_t>((work + pgrid - 1) / pgrid, kMinWarps,
                                                    (a.pull_div ? kPullThreads : kPushThreads) / 32);
        const unsigned ctas = static_cast<unsigned>(
            std::min<uint64_t>(pgrid, std::max<uint64_t>(1, (work + warps - 1) / warps)));
        void *kargs[] = {&a, &pg, &solve_state, &max_rounds};
        HYT_CUDA(cudaLaunchCooperativeKernel(solve, dim3(ctas), dim3(static_cast<unsigned>(32 * warps)), kargs,
                                             pull_smem, s));
    } else {
        HYT_CUDA(cudaMemcpyAsync(d_args, &a, sizeof(a), cudaMemcpyHostToDevice, s));
        HYT_CUDA(cudaMemcpyAsync(hdr, &h0, sizeof(h0), cudaMemcpyHostToDevice, s));
        sssp_init_kernel<<<grid_for(V, 256, 148 * 8), 256, 0, s>>>(d_args);
        HYT_CUDA(cudaGetLastError());
    }
    if (in_graph && far_pile) {
        if (!reuse) {
            cudaGraphNodeParams cp = {};
            cp.type = cudaGraphNodeTypeConditional;
            cp.conditional.handle = loop.cond;
            cp.conditional.type = cudaGraphCondTypeWhile;
            cp.conditional.size = 1;
            cudaGraphNode_t cnode;
            HYT_CUDA(cudaGraphAddNode(&cnode, loop.graph, nullptr, 0, &cp));
            cudaGraph_t body = cp.conditional.phGraph_out[0];
            void *kargs[] = {&d_args};
            cudaGraphNode_t prev = nullptr, node;
            auto add = [&](const void *f, dim3 gd, dim3 bd) {
                cudaKernelNodeParams kp = {};
                kp.func = const_cast<void *>(f);
                kp.gridDim = gd;
                kp.blockDim = bd;
                kp.kernelParams = kargs;
                HYT_CUDA(cudaGraphAddKernelNode(&node, body, prev ? &prev : nullptr, prev ? 1 : 0, &kp));
                prev = node;
            };
            add(reinterpret_cast<void *>(sssp_split_kernel), dim3(grid), dim3(kSSThreads));
            add(reinterpret_cast<void *>(sssp_expand_kernel<WK>), dim3(grid), dim3(kSSThreads));
            add(reinterpret_cast<void *>(sssp_hub_kernel<WK>), dim3(grid), dim3(kSSThreads));
            add(reinterpret_cast<void *>(sssp_round_end_kernel), dim3(1), dim3(1));
            HYT_CUDA(cudaGraphInstantiate(&loop.exec, loop.graph, 0));
            loop.set_key(&key, sizeof(key));
        }
        HYT_CUDA(cudaGraphLaunch(loop.exec, s));
    } else if (!persistent) {
        EventTimer kt;
        for (uint32_t r = 0; r < max_rounds; ++r) {
            if (flags & HYT_RUN_PROFILE) kt.start(s);
            if (far_pile) sssp_split_kernel<<<grid, kSSThreads, 0, s>>>(d_args);
            if (a.pull_div) {
                sssp_expand_kernel<WK, false, true><<<grid, kSSThreads, 0, s>>>(d_args);
                sssp_hub_kernel<WK, false, true><<<grid, kSSThreads, 0, s>>>(d_args);
                sssp_pull_kernel<WK, kPacked><<<pgrid, kPullThreads, pull_smem, s>>>(a, pg);
                sssp_round_close_kernel<<<1, 1, 0, s>>>(d_args);
            } else {
                sssp_expand_kernel<WK><<<grid, kSSThreads, 0, s>>>(d_args);
                sssp_hub_kernel<WK><<<grid, kSSThreads, 0, s>>>(d_args);
            }
            if (flags & HYT_RUN_PROFILE) kt.stop(s);
            if (!a.pull_div) sssp_round_end_kernel<<<1, 1, 0, s>>>(d_args);
            HYT_CUDA(cudaGetLastError());
            launches += per_round;
            hot += a.pull_div ? per_round : per_round - 1;
            uint32_t done = 0;
            HYT_CUDA(cudaMemcpyAsync(&done, &hdr->done, sizeof(done), cudaMemcpyDeviceToHost, s));
            HYT_CUDA(cudaStreamSynchronize(s));
            if (flags & HYT_RUN_PROFILE) kernel_ms += kt.ms();
            if (done) break;
        }
    }
    if (kPacked && !persistent && a.inf != HYT_DIST_INF_U32) {
        sssp_unreached_kernel<<<grid_for(V, 256, 148 * 8), 256, 0, s>>>(a.dist, a.V, a.inf);
        HYT_CUDA(cudaGetLastError());
    }
    SSHeader local{};
    SSHeader *hp = g.host_scratch.ptr ? reinterpret_cast<SSHeader *>(g.host_scratch.ptr) : &local;
    static_assert(sizeof(SSHeader) <= 64 * sizeof(uint64_t), "the header fits the pinned readback area");
    HYT_CUDA(cudaMemcpyAsync(hp, hdr, sizeof(SSHeader), cudaMemcpyDeviceToHost, s));
    total.stop(s);
    const double total_ms = total.ms();
    const SSHeader h = *hp;
    if (in_graph && far_pile) launches += per_round * h.round;
    if (h.error) fail(HYT_E_TIMEOUT, "SSSP: a bounded wait at a grid barrier ran out");
    if (dist_out) graph_emit(g, dist_out, g.dist.get(), s);
    if (stats) {
        stats->iterations = h.round;
        stats->converged = h.converged;
        stats->residual = 0.0;
        stats->device_ms = total_ms;
        stats->kernel_ms = kernel_ms;
        stats->kernel_launches = hot;
        stats->total_launches = launches;
        stats->edges_processed = h.relaxations;
        stats->vertices_processed = h.frontier_total;
        // per frontier vertex: 8 B offset pair (read twice) + 4 B label +
        // 4 B queue entry; per edge: 4 B column + 4 B weight + 4 B label.
        stats->algorithmic_bytes = 16ull * h.frontier_total + 12ull * h.relaxations;
    }
}

}  // namespace

uint32_t sssp_default_delta(const GraphImpl &g) {
    // Measured on R-MAT scale 24 (bucket widths 4 .. infinity): with batched
    // relaxations the extra rounds of narrow buckets cost more than the
    // relaxations they save, so the default is one bucket (frontier
    // Bellman-Ford).  Callers pick a finite width with params.delta; a
    // graph's 2x-mean-weight width is kept in g.default_delta for that.
    (void)g;
    return kNoDelta;
}

void sssp_run(GraphImpl &g, const hyt_sssp_params &p, uint32_t *dist_out, hyt_run_stats *stats) {
    if (!(g.flags & HYT_GRAPH_PUSH)) fail(HYT_E_INVALID, "graph was created without HYT_GRAPH_PUSH");
    if (p.source >= g.V) fail(HYT_E_INVALID, "SSSP source vertex is out of range");
    if (!g.weights_ok) fail(HYT_E_INVALID, "SSSP requires finite non-negative edge weights");
    cudaStream_t s = p.stream ? static_cast<cudaStream_t>(p.stream) : g.stream;
    // Termination is guaranteed (labels only decrease, weights >= 0); the
    // round cap is a safety bound on the device loop.
    const uint64_t cap = std::min<uint64_t>(4 * g.V + 1024, 0x7FFFFFFFull);
    const uint32_t max_rounds = p.max_rounds ? p.max_rounds : static_cast<uint32_t>(cap);
    const uint32_t delta = p.delta ? p.delta : sssp_default_delta(g);
    const uint32_t src = graph_vertex(g, p.source, s);
    switch (g.weight_kind) {
        case HYT_WEIGHTS_NONE: sssp_solve<HYT_WEIGHTS_NONE, false>(g, src, delta, max_rounds, p.flags, s, dist_out, stats); break;
        case HYT_WEIGHTS_U32:
            // sweeps run with one bucket only; other solves do not read the CSC
            if (g.in_pack_bits && delta == kNoDelta)
                sssp_solve<HYT_WEIGHTS_U32, true>(g, src, delta, max_rounds, p.flags, s, dist_out, stats);
            else
                sssp_solve<HYT_WEIGHTS_U32, false>(g, src, delta, max_rounds, p.flags, s, dist_out, stats);
            break;
        case HYT_WEIGHTS_F32: sssp_solve<HYT_WEIGHTS_F32, false>(g, src, kNoDelta, max_rounds, p.flags, s, dist_out, stats); break;
        default: fail(HYT_E_INTERNAL, "unknown weight kind");
    }
}

// Round loop of an out-of-HBM solve: per round the frontier's partition
// metrics go to the source, which places every partition's edges (resident,
// staged, mapped host memory) or compacts them; then the usual expansion.
template <int WK>
static void sssp_partitioned_solve(GraphImpl &g, PushSource &src, uint32_t source, uint32_t max_rounds,
                                   cudaStream_t s, uint32_t *dist_out, hyt_run_stats *stats) {
    const uint64_t V = g.V;
    const size_t P = src.parts();
    if (P == 0 || P > kMaxParts) fail(HYT_E_UNSUPPORTED, "partitioned SSSP supports 1..1024 partitions");
    if (g.dist.count < V) g.dist.allocate(V);
    if (g.stamp.count < 2 * V) g.stamp.allocate(2 * V);
    for (int i = 0; i < 2; ++i) {
        if (g.queue[i].count < V) g.queue[i].allocate(V);
        if (g.far[i].count < V) g.far[i].allocate(V);
    }
    const uint64_t hub_cap = V + g.E / kHubChunk + 2;
    if (g.hub_tasks.count < hub_cap) g.hub_tasks.allocate(hub_cap);
    const size_t sb = 512 + sizeof(SSHeader);
    if (g.sssp_state.count < sb) g.sssp_state.allocate(sb);
    SSArgs *d_args = reinterpret_cast<SSArgs *>(g.sssp_state.get());
    SSHeader *hdr = reinterpret_cast<SSHeader *>(g.sssp_state.get() + 256);
    DeviceArray<EdgeLoc> d_loc(P);
    DeviceArray<PartMetrics> d_metrics(P);
    DeviceArray<uint32_t> d_list(V + 1);
    uint32_t *d_count = d_list.get() + V;
    PinnedArray<uint32_t> h_list;

    SSArgs a{};
    a.row_off = g.row_offsets.get();
    a.dist = g.dist.get();
    a.stamp = g.stamp.get();
    a.fstamp = g.stamp.get() + V;
    for (int i = 0; i < 2; ++i) {
        a.queue[i] = g.queue[i].get();
        a.far[i] = g.far[i].get();
    }
    a.hubs = g.hub_tasks.get();
    a.hdr = hdr;
    a.V = static_cast<uint32_t>(V);
    a.source = source;
    a.inf = (WK == HYT_WEIGHTS_F32) ? 0x7F800000u : HYT_DIST_INF_U32;
    a.loc = d_loc.get();
    a.part_shift = src.part_shift();
    SSHeader h0{};
    h0.qsize[0] = 1;
    h0.max_rounds = max_rounds;
    h0.delta = kNoDelta;
    h0.threshold = 0xFFFFFFFFu;

    const int grid = expand_grid<WK>();
    EventTimer total;
    total.start(s);
    HYT_CUDA(cudaMemcpyAsync(d_args, &a, sizeof(a), cudaMemcpyHostToDevice, s));
    HYT_CUDA(cudaMemcpyAsync(hdr, &h0, sizeof(h0), cudaMemcpyHostToDevice, s));
    sssp_init_kernel<<<grid_for(V, 256, 148 * 8), 256, 0, s>>>(d_args);
    HYT_CUDA(cudaGetLastError());
    uint32_t launches = 1;
    std::vector<PartMetrics> metrics(P);
    RoundPlan plan;
    for (uint32_t r = 0; r < max_rounds; ++r) {
        sssp_split_kernel<<<grid, kSSThreads, 0, s>>>(d_args);
        HYT_CUDA(cudaMemsetAsync(d_metrics.get(), 0, P * sizeof(PartMetrics), s));
        sssp_part_stats_kernel<<<sm_count() * 2, kSSThreads, 0, s>>>(d_args, static_cast<uint32_t>(P), d_metrics.get());
        HYT_CUDA(cudaGetLastError());
        HYT_CUDA(cudaMemcpyAsync(metrics.data(), d_metrics.get(), P * sizeof(PartMetrics), cudaMemcpyDeviceToHost, s));
        HYT_CUDA(cudaStreamSynchronize(s));
        src.plan_round(metrics, plan);
        launches += 2;
        for (size_t w = 0; w < plan.waves.size(); ++w) {
            src.enter_wave(w, s);
            HYT_CUDA(cudaMemcpyAsync(d_loc.get(), plan.waves[w].data(), P * sizeof(EdgeLoc), cudaMemcpyHostToDevice,
                                     s));
            sssp_expand_kernel<WK, true><<<grid, kSSThreads, 0, s>>>(d_args);
            sssp_hub_kernel<WK, true><<<grid, kSSThreads, 0, s>>>(d_args);
            HYT_CUDA(cudaGetLastError());
            HYT_CUDA(cudaMemsetAsync(&hdr->hub_count, 0, sizeof(uint32_t), s));
            src.leave_wave(w, s);
            launches += 2;
        }
        if (plan.compacted) {
            HYT_CUDA(cudaMemsetAsync(d_count, 0, sizeof(uint32_t), s));
            sssp_compacted_list_kernel<<<grid_for(V, 256, 148 * 8), 256, 0, s>>>(d_args, d_list.get(), d_count);
            HYT_CUDA(cudaGetLastError());
            uint32_t n = 0;
            HYT_CUDA(cudaMemcpyAsync(&n, d_count, sizeof(n), cudaMemcpyDeviceToHost, s));
            HYT_CUDA(cudaStreamSynchronize(s));
            if (n) {
                if (h_list.count < n) h_list.allocate(std::max<size_t>(n, 1u << 20));
                HYT_CUDA(cudaMemcpyAsync(h_list.ptr, d_list.get(), n * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
                HYT_CUDA(cudaStreamSynchronize(s));
                const CompactPayload pk = src.compact(h_list.ptr, n, s);
                sssp_expand_packed_kernel<WK><<<grid, kSSThreads, 0, s>>>(d_args, pk);
                HYT_CUDA(cudaGetLastError());
                launches += 2;
            }
        }
        sssp_round_end_kernel<<<1, 1, 0, s>>>(d_args);
        HYT_CUDA(cudaGetLastError());
        ++launches;
        src.end_round(s);
        uint32_t done = 0;
        HYT_CUDA(cudaMemcpyAsync(&done, &hdr->done, sizeof(done), cudaMemcpyDeviceToHost, s));
        HYT_CUDA(cudaStreamSynchronize(s));
        if (done) break;
    }
    SSHeader h{};
    HYT_CUDA(cudaMemcpyAsync(&h, hdr, sizeof(h), cudaMemcpyDeviceToHost, s));
    total.stop(s);
    const double total_ms = total.ms();
    if (dist_out) copy_from_device(dist_out, g.dist.get(), V * sizeof(uint32_t), s);
    if (stats) {
        stats->iterations = h.round;
        stats->converged = h.converged;
        stats->device_ms = total_ms;
        stats->total_launches = launches;
        stats->edges_processed = h.relaxations;
        stats->vertices_processed = h.frontier_total;
        stats->algorithmic_bytes = 16ull * h.frontier_total + 12ull * h.relaxations;
    }
}

void sssp_partitioned(GraphImpl &g, PushSource &src, uint32_t source, uint32_t max_rounds, cudaStream_t s,
                      uint32_t *dist_out, hyt_run_stats *stats) {
    if (source >= g.V) fail(HYT_E_INVALID, "SSSP source vertex is out of range");
    if (!g.weights_ok) fail(HYT_E_INVALID, "SSSP requires finite non-negative edge weights");
    const uint64_t cap = std::min<uint64_t>(4 * g.V + 1024, 0x7FFFFFFFull);
    const uint32_t rounds = max_rounds ? max_rounds : static_cast<uint32_t>(cap);
    switch (g.weight_kind) {
        case HYT_WEIGHTS_NONE: sssp_partitioned_solve<HYT_WEIGHTS_NONE>(g, src, source, rounds, s, dist_out, stats); break;
        case HYT_WEIGHTS_U32: sssp_partitioned_solve<HYT_WEIGHTS_U32>(g, src, source, rounds, s, dist_out, stats); break;
        case HYT_WEIGHTS_F32: sssp_partitioned_solve<HYT_WEIGHTS_F32>(g, src, source, rounds, s, dist_out, stats); break;
        default: fail(HYT_E_INTERNAL, "unknown weight kind");
    }
}

}  // namespace hyt

namespace hyt {

// ===========================================================================
// SSSP that allocates nothing: hyt_sssp_noalloc (include/hyt/capi.h).
//
// For callers that cannot call cudaMalloc: a host application whose caching
// allocator already holds the device's free memory, a latency-critical loop
// that must not pay cudaMalloc's implicit device synchronisation, or a plugin
// host that forbids its components to allocate.  The caller passes its CSR
// and the output label array in device memory; every other buffer the solver
// needs lives in one file-scope __device__ array of kNoAllocScratchBytes that
// each GPU loading this library holds until the process exits.
//
// The first call on a device looks up the array's device address
// (cudaGetSymbolAddress) with that device current and caches it; make that
// first call before any stream capture.  Every call shares the array and it
// keeps the previous call's contents; whatever must start at zero is cleared
// by the call itself.  Calls whose work overlaps on the GPU (other streams,
// other threads) race on the array.
// ===========================================================================
namespace {

constexpr uint64_t kNoAllocMaxVertices = HYT_NOALLOC_MAX_VERTICES;
constexpr uint64_t kNoAllocMaxEdges = HYT_NOALLOC_MAX_EDGES;
constexpr uint64_t kNoAllocHubCap = kNoAllocMaxVertices + kNoAllocMaxEdges / kHubChunk + 2;
// args (256 B) | header (256 B) | check word (64 B) | stamp+fstamp u32[2V] |
// queue u32[2][V] | far u32[2][V] | hub tasks uint2[hub cap]
constexpr size_t kNoAllocHeadBytes = 1024;
// head: arguments at 0, header at 256, validation flags at 512
static_assert(sizeof(SSArgs) <= 256 && sizeof(SSHeader) <= 256, "no-alloc head layout");
constexpr size_t kNoAllocScratchBytes =
    kNoAllocHeadBytes + 6 * sizeof(uint32_t) * kNoAllocMaxVertices + sizeof(uint2) * kNoAllocHubCap;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
void *g_noalloc_address[kNoAllocMaxDevices] = {};

// Device address of the scratch array on the current device.  In host code
// the name g_noalloc_scratch is only a host-side stand-in, never passed to a
// kernel.
unsigned char *noalloc_scratch(int device) {
    if (device < 0 || device >= kNoAllocMaxDevices) fail(HYT_E_UNSUPPORTED, "hyt_sssp_noalloc: device ordinal too large");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_address[device]) {
        void *p = nullptr;
        HYT_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        g_noalloc_address[device] = p;
    }
    return static_cast<unsigned char *>(g_noalloc_address[device]);
}

// Rejects malformed CSR input before any kernel indexes with it.
__global__ void noalloc_check_kernel(const uint64_t *off, const uint32_t *cols, const uint32_t *w, uint32_t wkind,
                                     uint64_t V, uint64_t E, uint32_t *bad) {
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    const uint64_t i0 = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    uint32_t b = 0;
    for (uint64_t v = i0; v < V; v += stride)
        if (off[v + 1] < off[v]) b |= 1u;
    for (uint64_t e = i0; e < E; e += stride) {
        if (cols[e] >= V) b |= 2u;
        if (wkind == HYT_WEIGHTS_F32) {
            const float x = __uint_as_float(w[e]);
            if (!(x >= 0.0f) || isinf(x)) b |= 4u;
        }
    }
    if (i0 == 0 && (off[0] != 0 || off[V] != E)) b |= 1u;
    if (b) atomicOr(bad, b);
}

template <int WK>
void sssp_noalloc_solve(const hyt_csr &csr, uint32_t source, uint32_t *dist, cudaStream_t s, unsigned char *scratch,
                        hyt_run_stats *stats) {
    const uint64_t V = csr.num_vertices, E = csr.num_edges;
    SSArgs *d_args = reinterpret_cast<SSArgs *>(scratch);
    SSHeader *hdr = reinterpret_cast<SSHeader *>(scratch + 256);
    uint32_t *check = reinterpret_cast<uint32_t *>(scratch + 512);
    uint32_t *stamp = reinterpret_cast<uint32_t *>(scratch + kNoAllocHeadBytes);
    uint32_t *queue0 = stamp + 2 * kNoAllocMaxVertices;
    uint32_t *queue1 = queue0 + kNoAllocMaxVertices;
    uint32_t *far0 = queue1 + kNoAllocMaxVertices;
    uint32_t *far1 = far0 + kNoAllocMaxVertices;
    uint2 *hubs = reinterpret_cast<uint2 *>(far1 + kNoAllocMaxVertices);

    HYT_CUDA(cudaMemsetAsync(check, 0, sizeof(uint32_t), s));
    noalloc_check_kernel<<<grid_for(std::max(V, E), 256, 148 * 8), 256, 0, s>>>(
        csr.row_offsets, csr.column_indices, static_cast<const uint32_t *>(csr.weights), WK, V, E, check);
    HYT_CUDA(cudaGetLastError());
    uint32_t bad = 0;
    HYT_CUDA(cudaMemcpyAsync(&bad, check, sizeof(bad), cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaStreamSynchronize(s));
    if (bad & 1u) fail(HYT_E_INVALID, "hyt_sssp_noalloc: row offsets must start at 0, be non-decreasing and end at E");
    if (bad & 2u) fail(HYT_E_INVALID, "hyt_sssp_noalloc: column index contains an invalid destination vertex ID");
    if (bad & 4u) fail(HYT_E_INVALID, "SSSP requires finite non-negative edge weights");

    SSArgs a{};
    a.row_off = csr.row_offsets;
    a.cols = csr.column_indices;
    a.weights = static_cast<const uint32_t *>(csr.weights);
    a.dist = dist;
    a.stamp = stamp;
    a.fstamp = stamp + kNoAllocMaxVertices;
    a.queue[0] = queue0;
    a.queue[1] = queue1;
    a.far[0] = far0;
    a.far[1] = far1;
    a.hubs = hubs;
    a.hdr = hdr;
    a.V = static_cast<uint32_t>(V);
    a.source = source;
    a.inf = (WK == HYT_WEIGHTS_F32) ? 0x7F800000u : HYT_DIST_INF_U32;
    a.use_cond = 0;

    SSHeader h0{};  // every counter of the round state starts at zero
    h0.qsize[0] = 1;
    h0.delta = kNoDelta;
    h0.threshold = 0xFFFFFFFFu;
    const uint32_t max_rounds = static_cast<uint32_t>(4 * V + 1024);
    h0.max_rounds = max_rounds;

    const int grid = expand_grid<WK>();
    HYT_CUDA(cudaMemcpyAsync(d_args, &a, sizeof(a), cudaMemcpyHostToDevice, s));
    HYT_CUDA(cudaMemcpyAsync(hdr, &h0, sizeof(h0), cudaMemcpyHostToDevice, s));
    sssp_init_kernel<<<grid_for(V, 256, 148 * 8), 256, 0, s>>>(d_args);
    HYT_CUDA(cudaGetLastError());
    uint32_t launches = 2;
    for (uint32_t r = 0; r < max_rounds; ++r) {
        sssp_split_kernel<<<grid, kSSThreads, 0, s>>>(d_args);
        sssp_expand_kernel<WK><<<grid, kSSThreads, 0, s>>>(d_args);
        sssp_hub_kernel<WK><<<grid, kSSThreads, 0, s>>>(d_args);
        sssp_round_end_kernel<<<1, 1, 0, s>>>(d_args);
        HYT_CUDA(cudaGetLastError());
        launches += 4;
        uint32_t done = 0;
        HYT_CUDA(cudaMemcpyAsync(&done, &hdr->done, sizeof(done), cudaMemcpyDeviceToHost, s));
        HYT_CUDA(cudaStreamSynchronize(s));
        if (done) break;
    }
    SSHeader h{};
    HYT_CUDA(cudaMemcpyAsync(&h, hdr, sizeof(h), cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaStreamSynchronize(s));
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        stats->iterations = h.round;
        stats->converged = h.converged;
        stats->total_launches = launches;
        stats->edges_processed = h.relaxations;
        stats->vertices_processed = h.frontier_total;
        stats->algorithmic_bytes = 16ull * h.frontier_total + 12ull * h.relaxations;
    }
}

}  // namespace

void sssp_noalloc(const hyt_csr &csr, uint32_t source, uint32_t *dist_out, void *stream, hyt_run_stats *stats) {
    const uint64_t V = csr.num_vertices, E = csr.num_edges;
    if (V == 0) fail(HYT_E_INVALID, "SSSP requires at least one vertex");
    if (V > kNoAllocMaxVertices || E > kNoAllocMaxEdges)
        fail(HYT_E_INVALID, "hyt_sssp_noalloc: graph exceeds the fixed scratch capacity (at most " +
                                std::to_string(kNoAllocMaxVertices) + " vertices and " +
                                std::to_string(kNoAllocMaxEdges) + " edges); use hyt_sssp for larger graphs");
    if (source >= V) fail(HYT_E_INVALID, "SSSP source vertex is out of range");
    if (csr.weight_kind > HYT_WEIGHTS_F32) fail(HYT_E_INVALID, "unknown weight_kind");
    int device = 0;
    HYT_CUDA(cudaGetDevice(&device));
    // Every array is dereferenced by kernels on the current device: host
    // memory and another GPU's memory are refused before any launch
    // (column_indices and weights are read only when there are edges).
    const bool edges = E > 0, weights = edges && csr.weight_kind != HYT_WEIGHTS_NONE;
    const std::pair<const void *, const char *> arrays[] = {{csr.row_offsets, "row_offsets"},
                                                           {csr.column_indices, edges ? "column_indices" : nullptr},
                                                           {csr.weights, weights ? "weights" : nullptr},
                                                           {dist_out, "dist_out"}};
    for (const auto &[ptr, name] : arrays) {
        if (!name) continue;
        int owner = -1;
        const PointerPlace place = pointer_place(ptr, device, &owner);
        if (place == PointerPlace::kHost)
            fail(HYT_E_INVALID, std::string("hyt_sssp_noalloc: ") + name +
                                    " must be device memory of the current device (got host memory)");
        if (place == PointerPlace::kOtherDevice)
            fail(HYT_E_INVALID, std::string("hyt_sssp_noalloc: ") + name + " is device memory of GPU " +
                                    std::to_string(owner) + ", not of the current device " +
                                    std::to_string(device));
    }
    unsigned char *scratch = noalloc_scratch(device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (csr.weight_kind) {
        case HYT_WEIGHTS_NONE: sssp_noalloc_solve<HYT_WEIGHTS_NONE>(csr, source, dist_out, s, scratch, stats); break;
        case HYT_WEIGHTS_U32: sssp_noalloc_solve<HYT_WEIGHTS_U32>(csr, source, dist_out, s, scratch, stats); break;
        default: sssp_noalloc_solve<HYT_WEIGHTS_F32>(csr, source, dist_out, s, scratch, stats); break;
    }
}

}  // namespace hyt
