// Multi-source SSSP: up to 8 sources on one graph in one solve
// (hyt_sssp_multi).
//
// Every source keeps the single-source definition (hyt_sssp; the
// reference's sssp_cpu fixed point, src/algorithms/sssp.cpp:109-234): the
// labels are the unique shortest-path distances, reached by any
// label-correcting schedule, so each lane is bit-identical to hyt_sssp from
// its source.
//
// The 8 labels of a vertex sit together in one 32-byte row (lanes beyond
// the query count stay at infinity), so work is shared across the sources:
//   push round -- the union frontier (vertices whose label dropped in any
//                 lane) is expanded once; per out-edge one id, one weight
//                 and one 32-byte label row of the head, then an atomicMin
//                 only for lanes that improve.  Rows of >= kHubDegree edges
//                 become 512-edge warp tasks of a second kernel.
//   pull sweep -- when the frontier's out-edges exceed E / 4, every row
//                 takes, per lane, the minimum of d[u] + w over its
//                 in-edges: one id and one 32-byte label row per in-edge
//                 for all lanes, 1 to 32 edges of a row side by side, 4
//                 label rows in flight per thread.  A row is skipped when
//                 no in-edge can lower it in any lane: its label is at most
//                 (lowest label of the frontier in that lane + smallest
//                 weight).  Tile rows are written with plain stores (one
//                 writer per row during a sweep).
// A sweep used to walk short rows one lane per row and extend labels with
// saturation: 8 sources on R-MAT scale 20 / 24 took 1.98 / 8.74 ms, now 1.69 /
// 7.81 ms, before the changes noted at the sweep and at the loop's
// instantiation.
// Per edge the memory traffic is about that of one single-source
// relaxation, whatever the number of lanes; the rounds are those of the
// deepest source.  Rounds run as a CUDA-graph conditional while-loop.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "graph.cuh"
#include "scratch.cuh"
#include "solvers.cuh"
#include "sssp_core.cuh"

namespace hyt {
namespace {

using ssc::extend;
using ssc::kHubChunk;
using ssc::kHubDegree;

constexpr int kML = 8;             // labels per vertex row (32 bytes)
constexpr int kMSThreads = 256;    // push kernels
constexpr int kMPThreads = 640;    // pull sweep (one CTA per SM; 102 registers a thread)

struct MSHeader {
    uint32_t round, done, converged, pad0;
    uint32_t qsize[2];
    uint32_t hub_count;
    uint32_t max_rounds;
    unsigned long long relaxations;     // push: frontier out-edges; pull: in-edges of the rows not skipped
    unsigned long long frontier_total;  // frontier vertices expanded
    unsigned long long frontier_edges;  // out-edges of this round's frontier
    uint32_t pull_rounds, task_cursor;  // task_cursor: pull tasks handed out beyond the dealt ones
    unsigned long long frontier_edges_next;  // out-edges of the next frontier, summed by the kernels that fill it
    uint32_t fmin[kML];      // lowest label of this round's frontier, per lane
    uint32_t fmin_inv[kML];  // ~(lowest label of the next frontier)
};

struct MSArgs {
    const uint64_t *row_off;
    const uint32_t *cols;
    const uint32_t *weights;
    uint32_t *dist;  // [V][kML]
    uint32_t *stamp;
    uint32_t *queue[2];
    uint2 *hubs;
    MSHeader *hdr;
    uint32_t V, k, inf, use_cond;
    cudaGraphConditionalHandle cond;
    uint32_t pull_div;
    uint64_t num_edges;
    uint32_t sources[kML];
    // pull side (CSC, weights in CSC order, task list)
    const uint64_t *in_off;
    const uint32_t *in_src;
    const uint32_t *in_w;
    const uint32_t *hot_vertex;
    const LongRow *long_rows;
    const uint4 *tasks;
    const uint32_t *out_deg;
    uint64_t num_tasks, dealt;  // dealt: dealt_tasks
    uint32_t num_hot;
    uint32_t skip_rows;  // 1: sweeps skip rows whose labels no in-edge can lower
    uint32_t min_w;      // smallest edge weight (bit pattern; 1 when unweighted)
    uint32_t bits;       // packed words in in_w: bits of the source id
};

struct Row8 {
    uint32_t d[kML];
};

// Arithmetic of a solve's labels.  kBounded: no shortest path of the graph
// can reach a.inf ((V - 1) * largest weight < a.inf) and a.inf + any weight
// does not wrap, so a label is extended by one add, and an unreached source's
// candidate stays at or above a.inf and never lowers anything.  Otherwise
// labels saturate (extend) and unreached sources are tested for.  With 8
// labels per edge the difference is a third of a sweep's instructions.
template <int WK, bool kBounded>
__device__ __forceinline__ uint32_t candidate(uint32_t d, uint32_t w, uint32_t inf) {
    if constexpr (WK == HYT_WEIGHTS_F32) {
        return extend<WK>(d, w);  // infinity stays infinity
    } else if constexpr (kBounded) {
        return d + w;
    } else {
        return d == inf ? inf : extend<WK>(d, w);
    }
}

// min(m, candidate(d, w)).
template <int WK, bool kBounded>
__device__ __forceinline__ uint32_t lower_by(uint32_t m, uint32_t d, uint32_t w, uint32_t inf) {
    if constexpr (kBounded && WK != HYT_WEIGHTS_F32) {
        return __viaddmin_u32(d, w, m);  // one instruction
    } else {
        return min(m, candidate<WK, kBounded>(d, w, inf));
    }
}

__device__ __forceinline__ Row8 load_row(const uint32_t *dist, uint32_t v) {
    const uint4 *p = reinterpret_cast<const uint4 *>(dist + size_t(v) * kML);
    const uint4 a = __ldcg(p), b = __ldcg(p + 1);
    return Row8{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}

__device__ __forceinline__ bool pull_round(const MSArgs &a) {
    if (!a.pull_div) return false;
    const unsigned long long fe = *(volatile const unsigned long long *)&a.hdr->frontier_edges;
    return fe * a.pull_div > a.num_edges;
}

struct View {
    uint32_t r, qn, next_stamp;
    const uint32_t *q;
    uint32_t *qnext, *qnext_size;
};

__device__ __forceinline__ View view(const MSArgs &a) {
    View w;
    w.r = *(volatile const uint32_t *)&a.hdr->round;
    const uint32_t odd = w.r & 1;
    w.qn = *(volatile const uint32_t *)(odd ? &a.hdr->qsize[1] : &a.hdr->qsize[0]);
    w.q = odd ? a.queue[1] : a.queue[0];
    w.qnext = odd ? a.queue[0] : a.queue[1];
    w.qnext_size = odd ? &a.hdr->qsize[0] : &a.hdr->qsize[1];
    w.next_stamp = w.r + 1;
    return w;
}

// What the next round needs to know of its frontier, gathered while it is
// filled: its out-edges and, in lane l < kML of the warp, the lowest label of
// lane l.
struct Gain {
    unsigned long long edges = 0;
    uint32_t low = 0xFFFFFFFFu;
};

// Notes the labels `now` of the lanes in `lower` (a bit mask, 0 in threads
// that lowered none); all 32 lanes.
__device__ __forceinline__ void note_lower(Gain &g, const Row8 &now, uint32_t lower, int lane) {
    uint32_t any = __reduce_or_sync(0xffffffffu, lower);
#pragma unroll
    for (int l = 0; l < kML; ++l) {
        if (!((any >> l) & 1u)) continue;
        const uint32_t t = __reduce_min_sync(0xffffffffu, ((lower >> l) & 1u) ? now.d[l] : 0xFFFFFFFFu);
        if (lane == l) g.low = min(g.low, t);
    }
}

__device__ __forceinline__ void flush_gain(const MSArgs &a, Gain &g, int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g.edges += __shfl_xor_sync(0xffffffffu, g.edges, o);
    if (lane == 0 && g.edges) atomicAdd(&a.hdr->frontier_edges_next, g.edges);
    if (lane < kML && g.low != 0xFFFFFFFFu) atomicMax(&a.hdr->fmin_inv[lane], ~g.low);
}

// Relaxes edge (u -> v, weight w) in every lane with u's labels du; true
// when some lane of v improved and v joins the next frontier now.  c gets the
// candidates, `lower` the lanes that improved.
template <int WK, bool kB>
__device__ __forceinline__ bool relax_row(const MSArgs &a, const View &w, const Row8 &du, uint32_t v, uint32_t wt,
                                          Row8 &c, uint32_t &lower) {
    const Row8 dv = load_row(a.dist, v);
#pragma unroll
    for (int l = 0; l < kML; ++l) {
        if (l >= static_cast<int>(a.k)) continue;
        c.d[l] = candidate<WK, kB>(du.d[l], wt, a.inf);
        if (c.d[l] < dv.d[l] && c.d[l] < atomicMin(a.dist + size_t(v) * kML + l, c.d[l])) lower |= 1u << l;
    }
    return lower && atomicExch(a.stamp + v, w.next_stamp) != w.next_stamp;
}

__global__ void ms_init_kernel(const MSArgs *__restrict__ args) {
    const MSArgs a = *args;
    const uint64_t n = uint64_t(a.V) * kML, stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += stride) a.dist[i] = a.inf;
    for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < a.V; v += stride) a.stamp[v] = ~0u;
}

// Sources: label 0 in their lane; each distinct source once in the first
// frontier.
__global__ void ms_sources_kernel(const MSArgs *__restrict__ args) {
    const MSArgs a = *args;
    if (threadIdx.x != 0) return;
    uint32_t n = 0;
    for (uint32_t l = 0; l < a.k; ++l) {
        const uint32_t s = a.sources[l];
        a.dist[size_t(s) * kML + l] = 0u;
        bool seen = false;
        for (uint32_t j = 0; j < l; ++j) seen |= a.sources[j] == s;
        if (!seen) {
            a.queue[0][n++] = s;
            a.stamp[s] = 0u;
            a.hdr->frontier_edges += a.row_off[s + 1] - a.row_off[s];  // round 0's frontier
        }
    }
    a.hdr->qsize[0] = n;
}


// Push round: a warp takes 32 frontier vertices; rows shorter than
// kHubDegree are walked as one combined edge list (each lane finds its
// edge's owner by a shuffle binary search and receives the owner's label
// row by shuffles), longer rows become hub tasks.
template <int WK, bool kB>
__global__ void __launch_bounds__(kMSThreads) ms_expand_kernel(const MSArgs *__restrict__ args) {
    const MSArgs a = *args;
    if (*(volatile uint32_t *)&a.hdr->done || pull_round(a)) return;
    const View w = view(a);
    const int lane = threadIdx.x & 31;
    const uint32_t gwarp = (blockIdx.x * kMSThreads + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * kMSThreads) >> 5;
    unsigned long long relaxed = 0;
    Gain gain;
    for (uint32_t base0 = gwarp * 32; base0 < w.qn; base0 += nwarps * 32) {
        const uint32_t i = base0 + lane;
        uint32_t deg = 0, u = 0;
        uint64_t off = 0;
        Row8 du;
#pragma unroll
        for (int l = 0; l < kML; ++l) du.d[l] = a.inf;
        if (i < w.qn) {
            u = w.q[i];
            off = a.row_off[u];
            const uint64_t full = a.row_off[u + 1] - off;
            relaxed += full;
            if (full >= kHubDegree) {
                const uint32_t nch = static_cast<uint32_t>((full + kHubChunk - 1) / kHubChunk);
                const uint32_t hb = atomicAdd(&a.hdr->hub_count, nch);
                for (uint32_t c = 0; c < nch; ++c) a.hubs[hb + c] = make_uint2(u, c);
            } else {
                deg = static_cast<uint32_t>(full);
                du = load_row(a.dist, u);
            }
        }
        uint32_t incl = deg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
        for (uint32_t b = 0; b < total; b += 32) {
            const uint32_t j = b + lane;
            uint32_t lo = 0;
#pragma unroll
            for (uint32_t step = 16; step > 0; step >>= 1) {
                const uint32_t probe = __shfl_sync(0xffffffffu, incl, lo + step - 1);
                if (probe <= j) lo += step;
            }
            const uint32_t o_incl = __shfl_sync(0xffffffffu, incl, lo);
            const uint32_t o_deg = __shfl_sync(0xffffffffu, deg, lo);
            const uint64_t o_off = __shfl_sync(0xffffffffu, off, lo);
            Row8 ou;
#pragma unroll
            for (int l = 0; l < kML; ++l) ou.d[l] = __shfl_sync(0xffffffffu, du.d[l], lo);
            bool join = false;
            uint32_t v = 0, lower = 0;
            Row8 c{};
            if (j < total) {
                const uint64_t e = o_off + (j - (o_incl - o_deg));
                v = dev::ld_stream(a.cols + e);
                join = relax_row<WK, kB>(a, w, ou, v, ssc::edge_weight<WK>(a.weights, e), c, lower);
            }
            if (a.pull_div) {
                note_lower(gain, c, lower, lane);
                if (join) gain.edges += a.out_deg[v];
            }
            const uint32_t vals[1] = {v};
            ssc::warp_append<1>(w.qnext, w.qnext_size, vals, join ? 1u : 0u, lane);
        }
    }
    if (a.pull_div) flush_gain(a, gain, lane);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) relaxed += __shfl_xor_sync(0xffffffffu, relaxed, o);
    if (lane == 0 && relaxed) atomicAdd(&a.hdr->relaxations, relaxed);
}

// One warp per kHubChunk-edge slice of a long frontier row.
template <int WK, bool kB>
__global__ void __launch_bounds__(kMSThreads) ms_hub_kernel(const MSArgs *__restrict__ args) {
    const MSArgs a = *args;
    if (*(volatile uint32_t *)&a.hdr->done || pull_round(a)) return;
    const View w = view(a);
    const uint32_t n = *(volatile uint32_t *)&a.hdr->hub_count;
    const int lane = threadIdx.x & 31;
    const uint32_t gwarp = (blockIdx.x * kMSThreads + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * kMSThreads) >> 5;
    Gain gain;
    for (uint32_t t = gwarp; t < n; t += nwarps) {
        const uint2 h = a.hubs[t];
        const uint64_t rb = a.row_off[h.x], re = a.row_off[h.x + 1];
        const uint64_t b = rb + uint64_t(h.y) * kHubChunk;
        const uint32_t len = static_cast<uint32_t>(((b + kHubChunk < re) ? b + kHubChunk : re) - b);
        const Row8 du = load_row(a.dist, h.x);
        for (uint32_t x = 0; x < len; x += 32) {
            bool join = false;
            uint32_t v = 0, lower = 0;
            Row8 c{};
            if (x + lane < len) {
                const uint64_t e = b + x + lane;
                v = dev::ld_stream(a.cols + e);
                join = relax_row<WK, kB>(a, w, du, v, ssc::edge_weight<WK>(a.weights, e), c, lower);
            }
            if (a.pull_div) {
                note_lower(gain, c, lower, lane);
                if (join) gain.edges += a.out_deg[v];
            }
            const uint32_t vals[1] = {v};
            ssc::warp_append<1>(w.qnext, w.qnext_size, vals, join ? 1u : 0u, lane);
        }
    }
    if (a.pull_div) flush_gain(a, gain, lane);
}

// ---- pull sweeps ------------------------------------------------------------
//
// Labels are read live (not snapshotted): rows lowered earlier in the same
// sweep -- the hub rows, whose chunks come first -- feed the rows after them.
// A minimum does not mind an edge taken twice, so threads without an edge of
// their own repeat their row's last one (the same sector) in place of
// predicated loads.
//
// A sweep waits for L2: a step's ids, then its labels, with 20 to 24 warps an
// SM to hide them (31 % of issue slots used, 0.3 of 1.0 sectors a clock).  So
// the next step's ids are loaded while this step's labels are on their way,
// at 640 threads for the registers that takes (768 spill, 512 hide less).  Eight
// sources on 1 M vertices, 15 M edges 1.66 -> 1.57 ms (768 threads 1.66, 512
// 1.62; 512 with 8 edges in flight 1.62); five on 2 M in input order 3.22 ->
// 3.09 (3.14, 3.36; 3.61).

constexpr int kPullN = 4;                  // edges in flight per thread
constexpr uint32_t kWideRow = 16 * kPullN;  // rows with this many in-edges are taken by the whole warp

// In-edges of one task, addressed relative to its first edge.
struct InEdges {
    const uint32_t *src, *w, *s_hot;  // ids and weights, or w: packed words (no hot slots)
    const uint32_t *dist;
    uint32_t inf, bits;
};

// kPullN edges' ids and weights as they were loaded (packed: `u` holds the
// words, decoded when they are used).
struct Edges {
    uint32_t u[kPullN], wt[kPullN];
};

// Edges b, b + step, ..., capped at edge `last`.
template <int WK, bool kB>
__device__ __forceinline__ void load_edges(const InEdges &E, uint32_t b, uint32_t last, uint32_t step, Edges &x) {
    constexpr bool kPacked = kB && WK == HYT_WEIGHTS_U32;
    const uint32_t *ids = kPacked ? E.w : E.src;
#pragma unroll
    for (int j = 0; j < kPullN; ++j) x.u[j] = dev::ld_stream(ids + min(b + j * step, last));
    if constexpr (!kPacked) {
#pragma unroll
        for (int j = 0; j < kPullN; ++j) x.wt[j] = ssc::edge_weight<WK>(E.w, min(b + j * step, last));
    }
}

// Minimum of the candidates of edges x (all their labels are loaded before the
// first is used) into m; then() runs while the labels are on their way.
template <int WK, bool kB, class F>
__device__ __forceinline__ void edges_min(const InEdges &E, const Edges &x, Row8 &m, F then) {
    constexpr bool kPacked = kB && WK == HYT_WEIGHTS_U32;
    const uint32_t mask = (1u << E.bits) - 1u;
    uint32_t wt[kPullN];
    Row8 du[kPullN];
#pragma unroll
    for (int j = 0; j < kPullN; ++j) {
        uint32_t u;
        if constexpr (kPacked) {
            u = x.u[j] & mask;
            wt[j] = x.u[j] >> E.bits;
        } else {
            u = x.u[j];
            wt[j] = x.wt[j];
            if (u & kHotTag) u = E.s_hot[u & ~kHotTag];
        }
        // the whole 32-byte row in one load: one L1 access per edge (two
        // 16-byte loads took the sector twice)
        asm volatile("ld.global.L2::evict_last.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(du[j].d[0]), "=r"(du[j].d[1]), "=r"(du[j].d[2]), "=r"(du[j].d[3]), "=r"(du[j].d[4]),
                       "=r"(du[j].d[5]), "=r"(du[j].d[6]), "=r"(du[j].d[7])
                     : "l"(E.dist + size_t(u) * kML));
    }
    then();
#pragma unroll
    for (int j = 0; j < kPullN; ++j)
#pragma unroll
        for (int l = 0; l < kML; ++l) m.d[l] = lower_by<WK, kB>(m.d[l], du[j].d[l], wt[j], E.inf);
}

// Lowest candidates over edges [b, e), b < e, by the whole warp; every lane
// returns them.
template <int WK, bool kB>
__device__ __forceinline__ Row8 span_min(const InEdges &E, uint32_t b, uint32_t e, int lane) {
    Row8 m;
#pragma unroll
    for (int l = 0; l < kML; ++l) m.d[l] = E.inf;
    Edges x;
    load_edges<WK, kB>(E, b + lane, e - 1, 32, x);
    for (uint32_t at = b; at < e; at += 32 * kPullN) {
        Edges nx;
        edges_min<WK, kB>(E, x, m, [&] { load_edges<WK, kB>(E, at + 32 * kPullN + lane, e - 1, 32, nx); });
        x = nx;
    }
#pragma unroll
    for (int l = 0; l < kML; ++l) m.d[l] = __reduce_min_sync(0xffffffffu, m.d[l]);
    return m;
}

// Lowest candidates of the warp's 32 rows (lane l: edges [lo, hi)), `slots`
// edges of a row side by side, 32 / slots rows a step; rows have at most
// slots * kPullN in-edges.  Rows without edges get an arbitrary result.  The
// next step's edges are loaded while this step's labels are on their way.
template <int WK, bool kB>
__device__ __forceinline__ Row8 group_min(const InEdges &E, uint32_t lo, uint32_t hi, int slots, int lane) {
    const int rows = 32 / slots;
    const uint32_t live = __ballot_sync(0xffffffffu, hi > lo);  // not 0
    Row8 mine;
#pragma unroll
    for (int l = 0; l < kML; ++l) mine.d[l] = E.inf;
    // steps without a row that has edges are left out
    const uint32_t step = rows == 32 ? 0xFFFFFFFFu : (1u << rows) - 1u;
    auto load = [&](int first, Edges &x) {
        const int owner = first + lane / slots;
        const uint32_t b = __shfl_sync(0xffffffffu, lo, owner);
        const uint32_t e = __shfl_sync(0xffffffffu, hi, owner);
        load_edges<WK, kB>(E, b + lane % slots, e > b ? e - 1 : 0u, slots, x);
    };
    int first = (__ffs(live) - 1) & ~(rows - 1);
    Edges x;
    load(first, x);
    for (;;) {
        const uint32_t rest = live & ~(step << first) & ~((1u << first) - 1u);
        const int next = rest ? (__ffs(rest) - 1) & ~(rows - 1) : 32;
        Edges nx;
        Row8 m;
#pragma unroll
        for (int l = 0; l < kML; ++l) m.d[l] = E.inf;
        edges_min<WK, kB>(E, x, m, [&] { if (next < 32) load(next, nx); });
        for (int o = 1; o < slots; o <<= 1)
#pragma unroll
            for (int l = 0; l < kML; ++l) m.d[l] = min(m.d[l], __shfl_xor_sync(0xffffffffu, m.d[l], o));
        const int from = ((lane - first) & (rows - 1)) * slots;
        const bool own = lane >= first && lane < first + rows;
#pragma unroll
        for (int l = 0; l < kML; ++l) {
            const uint32_t t = __shfl_sync(0xffffffffu, m.d[l], from);
            if (own) mine.d[l] = t;
        }
        if (next >= 32) break;
        first = next;
        x = nx;
    }
    return mine;
}

// Lowers row r's labels to m (lanes that improve); true when r joins the
// next frontier now.  Long rows: every chunk of the row may lower it.
__device__ __forceinline__ bool pull_lower(const MSArgs &a, const View &w, uint32_t r, const Row8 &m, uint32_t &lower) {
    const Row8 cur = load_row(a.dist, r);
#pragma unroll
    for (int l = 0; l < kML; ++l)
        if (l < static_cast<int>(a.k) && m.d[l] < cur.d[l] && m.d[l] < atomicMin(a.dist + size_t(r) * kML + l, m.d[l]))
            lower |= 1u << l;
    return lower && atomicExch(a.stamp + r, w.next_stamp) != w.next_stamp;
}

// True when no in-edge can lower row labels `cur` in any lane this round.
__device__ __forceinline__ bool row_settled(const MSArgs &a, const uint32_t *s_skip, const Row8 &cur) {
    bool settled = true;
#pragma unroll
    for (int l = 0; l < kML; ++l)
        if (l < static_cast<int>(a.k)) settled &= cur.d[l] <= s_skip[l];
    return settled;
}

template <int WK, bool kB>
__global__ void __launch_bounds__(kMPThreads, 1) ms_pull_kernel(const MSArgs *__restrict__ args) {
    extern __shared__ __align__(16) uint32_t s_hot[];  // vertex ids of the hot slots
    __shared__ uint32_t s_skip[kML];
    const MSArgs a = *args;
    if (*(volatile uint32_t *)&a.hdr->done || !pull_round(a)) return;
    const View w = view(a);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < a.num_hot; i += blockDim.x) s_hot[i] = a.hot_vertex[i];
    if (threadIdx.x < kML) {
        // an in-edge lowers lane l only from a source whose label of that
        // lane dropped last round; a lane without any cannot improve
        const uint32_t f = *(volatile const uint32_t *)&a.hdr->fmin[threadIdx.x];
        s_skip[threadIdx.x] = f < a.inf ? extend<WK>(f, a.min_w) : 0xFFFFFFFFu;
    }
    __syncthreads();
    const uint64_t nwarps = uint64_t(gridDim.x) * (kMPThreads / 32);
    constexpr bool kPacked = kB && WK == HYT_WEIGHTS_U32;
    const uint32_t *pf_a = kPacked ? a.in_w : a.in_src;
    const uint32_t *pf_w = (kPacked || WK == HYT_WEIGHTS_NONE) ? nullptr : a.in_w;
    InEdges E{nullptr, nullptr, s_hot, a.dist, a.inf, a.bits};
    unsigned long long relaxed = 0;  // in-edges relaxed (chunks counted by lane 0, tile rows by their lanes)
    Gain gain;
    const uint64_t dealt = max(a.dealt, min(a.num_tasks, nwarps));
    uint64_t task = uint64_t(blockIdx.x) * (kMPThreads / 32) + warp;
    uint4 d = task < a.num_tasks ? a.tasks[task] : make_uint4(0, 0, 0, 0);
    while (task < a.num_tasks) {
        uint64_t next = task + nwarps;
        uint32_t ticket = 0;
        const bool ask = next >= dealt;
        if (ask && lane == 0) ticket = atomicAdd(&a.hdr->task_cursor, 1u);
        uint4 nd = ask ? make_uint4(0, 0, 0, 0) : a.tasks[next];
        const uint64_t e0 = task_first_edge(d);
        E.src = a.in_src + e0;
        E.w = (WK == HYT_WEIGHTS_NONE) ? nullptr : a.in_w + e0;
        if (!ask) prefetch_task(nd, pf_a, pf_w, lane);
        if (task_is_chunk(d)) {
            const uint32_t r = a.long_rows[d.z].row, n = task_edges(d);
            uint32_t settled = 0;
            if (lane == 0 && a.skip_rows) settled = row_settled(a, s_skip, load_row(a.dist, r));
            if (!__shfl_sync(0xffffffffu, settled, 0)) {
                const Row8 m = span_min<WK, kB>(E, 0, n, lane);
                uint32_t lower = 0;
                if (lane == 0) {
                    relaxed += n;
                    if (pull_lower(a, w, r, m, lower)) {
                        gain.edges += a.out_deg[r];
                        ssc::append(w.qnext, w.qnext_size, r);
                    }
                }
                note_lower(gain, m, lower, lane);
            }
        } else {
            for (uint32_t rb = d.z; rb < d.w; rb += 32) {
                const uint32_t r = rb + lane;
                uint32_t lo = 0, hi = 0;
                Row8 cur{};
                if (r < d.w) {
                    lo = static_cast<uint32_t>(a.in_off[r] - e0);
                    hi = static_cast<uint32_t>(a.in_off[r + 1] - e0);
                    if (hi > lo) {
                        cur = load_row(a.dist, r);
                        if (a.skip_rows && row_settled(a, s_skip, cur)) hi = lo;
                    }
                }
                relaxed += hi - lo;
                const bool wide = hi - lo >= kWideRow;
                const uint32_t hs = wide ? lo : hi;  // group steps see a wide row as empty
                const uint32_t most = __reduce_max_sync(0xffffffffu, hs - lo);
                const uint32_t big = __ballot_sync(0xffffffffu, wide);
                if (!most && !big) continue;
                Row8 m;
#pragma unroll
                for (int l = 0; l < kML; ++l) m.d[l] = a.inf;
                // the fewest slots a row that hold its edges in one round of loads
                if (most) m = group_min<WK, kB>(E, lo, hs, most > 32 ? 16 : most > 16 ? 8 : most > 8 ? 4 : most > 4 ? 2 : 1, lane);
                for (uint32_t b = big; b; b &= b - 1) {
                    const int o = __ffs(b) - 1;
                    const Row8 t = span_min<WK, kB>(E, __shfl_sync(0xffffffffu, lo, o), __shfl_sync(0xffffffffu, hi, o), lane);
                    if (lane == o) m = t;
                }
                // a tile row has exactly one writer during a sweep (the warp
                // that owns its tile) and no push runs beside a sweep: plain stores
                uint32_t lower = 0;
                if (hi > lo) {
#pragma unroll
                    for (int l = 0; l < kML; ++l)
                        if (l < static_cast<int>(a.k) && m.d[l] < cur.d[l]) {
                            cur.d[l] = m.d[l];
                            lower |= 1u << l;
                        }
                    if (lower) {
                        uint4 *p = reinterpret_cast<uint4 *>(a.dist + size_t(r) * kML);
                        p[0] = make_uint4(cur.d[0], cur.d[1], cur.d[2], cur.d[3]);
                        p[1] = make_uint4(cur.d[4], cur.d[5], cur.d[6], cur.d[7]);
                        a.stamp[r] = w.next_stamp;
                        gain.edges += a.out_deg[r];
                    }
                }
                note_lower(gain, cur, lower, lane);
                const uint32_t vals[1] = {r};
                ssc::warp_append<1>(w.qnext, w.qnext_size, vals, lower ? 1u : 0u, lane);
            }
        }
        if (ask) {
            next = dealt + __shfl_sync(0xffffffffu, ticket, 0);
            if (next < a.num_tasks) nd = a.tasks[next];
        }
        task = next;
        d = nd;
    }
    flush_gain(a, gain, lane);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) relaxed += __shfl_xor_sync(0xffffffffu, relaxed, o);
    if (lane == 0 && relaxed) atomicAdd(&a.hdr->relaxations, relaxed);
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.hdr->pull_rounds, 1u);
}

// Round-end bookkeeping (one thread): true when the solve is finished.
__device__ __forceinline__ bool ms_end_round(const MSArgs &a, MSHeader *h) {
    const uint32_t r = h->round;
    const uint32_t n_next = h->qsize[(r + 1) & 1];
    h->frontier_total += h->qsize[r & 1];
    h->qsize[r & 1] = 0;
    h->hub_count = 0;
    h->frontier_edges = 0;
    h->round = r + 1;
    const bool conv = n_next == 0;
    if (conv || r + 1 >= h->max_rounds) {
        h->done = 1;
        h->converged = conv ? 1u : 0u;
        if (a.use_cond) cudaGraphSetConditional(a.cond, 0);
        return true;
    }
    return false;
}

__global__ void ms_round_end_kernel(const MSArgs *__restrict__ args) {
    const MSArgs a = *args;
    MSHeader *h = a.hdr;
    if (h->done) return;
    ms_end_round(a, h);
}

// End of a round of a pull-capable solve (one thread): the round's kernels
// have summed the next frontier's out-edges (the next round's push / pull
// decision) and found its lowest labels.
__global__ void ms_round_close_kernel(const MSArgs *__restrict__ args) {
    const MSArgs a = *args;
    MSHeader *h = a.hdr;
    if (h->done) return;
    const unsigned long long fe = h->frontier_edges_next;
    h->frontier_edges_next = 0;
    h->task_cursor = 0;
#pragma unroll
    for (int l = 0; l < kML; ++l) {
        h->fmin[l] = ~h->fmin_inv[l];  // all ones when no label of the lane dropped
        h->fmin_inv[l] = 0;
    }
    ms_end_round(a, h);
    h->frontier_edges = fe;
}

// out[l][c] = dist[inv[c]][l] (caller order c; inv NULL: identity); labels of
// unreached vertices (inf or above) become `unreached`.
__global__ void ms_emit_kernel(const uint32_t *__restrict__ dist, const uint32_t *__restrict__ inv, uint64_t V,
                               uint32_t k, uint32_t inf, uint32_t unreached, uint32_t *__restrict__ out) {
    for (uint64_t c = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; c < V; c += uint64_t(gridDim.x) * blockDim.x) {
        const uint32_t v = inv ? inv[c] : static_cast<uint32_t>(c);
        const Row8 r = load_row(dist, v);
        for (uint32_t l = 0; l < k; ++l) out[l * V + c] = r.d[l] < inf ? r.d[l] : unreached;
    }
}

template <int WK, bool kB>
int ms_push_grid() {
    static int g = 0;
    if (g == 0) {
        int per_sm = 0;
        HYT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ms_expand_kernel<WK, kB>, kMSThreads, 0));
        g = sm_count() * std::max(per_sm, 1);
    }
    return g;
}

template <int WK, bool kB>
void ms_solve(GraphImpl &g, const uint32_t *sources, uint32_t k, uint32_t max_rounds, uint32_t flags, cudaStream_t s,
              uint32_t max_w, uint32_t *out, hyt_run_stats *stats) {
    const uint64_t V = g.V;
    if (g.ms_dist.count < V * kML) g.ms_dist.allocate(V * kML);
    if (g.stamp.count < 2 * V) g.stamp.allocate(2 * V);
    for (int i = 0; i < 2; ++i)
        if (g.queue[i].count < V) g.queue[i].allocate(V);
    const uint64_t hub_cap = V + g.E / kHubChunk + 2;
    if (g.hub_tasks.count < hub_cap) g.hub_tasks.allocate(hub_cap);
    const size_t sb = 512 + sizeof(MSHeader);
    if (g.ms_state.count < sb) g.ms_state.allocate(sb);
    MSArgs *d_args = reinterpret_cast<MSArgs *>(g.ms_state.get());
    MSHeader *hdr = reinterpret_cast<MSHeader *>(g.ms_state.get() + 512);
    static_assert(sizeof(MSArgs) <= 512, "MSArgs must fit its 512-byte slot");

    MSArgs a{};
    a.row_off = g.row_offsets.get();
    a.cols = g.cols.get();
    a.weights = g.weights.get();
    a.dist = g.ms_dist.get();
    a.stamp = g.stamp.get();
    a.queue[0] = g.queue[0].get();
    a.queue[1] = g.queue[1].get();
    a.hubs = g.hub_tasks.get();
    a.hdr = hdr;
    a.V = static_cast<uint32_t>(V);
    a.k = k;
    const uint32_t unreached = (WK == HYT_WEIGHTS_F32) ? 0x7F800000u : HYT_DIST_INF_U32;
    a.inf = kB ? HYT_DIST_INF_U32 - max_w : unreached;
    a.num_edges = g.E;
    for (uint32_t l = 0; l < k; ++l) a.sources[l] = graph_vertex(g, sources[l], s);
    const bool pull_ok = (g.flags & HYT_GRAPH_PULL) && (WK == HYT_WEIGHTS_NONE || g.in_weights.get()) && g.E > 0 &&
                         g.pull_tasks.get() && size_t(g.num_hot) * 4 <= kPRSmemMax;
    a.pull_div = pull_ok ? 4u : 0u;
    if (pull_ok) {
        a.in_off = g.in_offsets.get();
        a.in_src = g.in_sources.get();
        a.in_w = g.in_weights.get();
        a.hot_vertex = g.hot_vertex.get();
        a.long_rows = g.long_rows.get();
        a.tasks = g.pull_tasks.get();
        a.num_tasks = g.num_chunks + g.num_tiles;
        a.dealt = dealt_tasks(g);
        a.bits = g.in_pack_bits;
        a.num_hot = a.bits ? 0u : g.num_hot;
    }
    if (pull_ok) {
        a.out_deg = g.out_degree.get();
        a.skip_rows = sssp_pull_skip() ? 1u : 0u;
        if (a.skip_rows) a.min_w = (WK == HYT_WEIGHTS_NONE) ? 1u : g.weight_range.low;
    }
    const unsigned pull_smem = static_cast<unsigned>(a.num_hot * sizeof(uint32_t));
    static bool attr = false;
    if (!attr) {
        HYT_CUDA(cudaFuncSetAttribute(ms_pull_kernel<WK, kB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kPRSmemMax)));
        attr = true;
    }
    const int grid = ms_push_grid<WK, kB>();
    const int pgrid = sm_count();

    MSHeader h0{};
    h0.max_rounds = max_rounds;
    const bool use_graph = !(flags & HYT_RUN_NO_GRAPH) && !(flags & HYT_RUN_PROFILE);
    // The round loop's kernels read everything through d_args, so its
    // instantiation, kept with the graph object, serves every solve of the same
    // shape (built on each call it cost 250 us: eight sources on 1 M vertices
    // 1.62 -> 1.36 ms, on 50 K 0.71 -> 0.46 ms).
    const struct {
        MSArgs *args;
        int wk, bounded, grid, pull_grid;
        unsigned smem, pull_div;
    } key{d_args, int(WK), int(kB), grid, pgrid, pull_smem, a.pull_div};
    static_assert(sizeof(key) == 32, "no padding: compared as bytes");
    LoopGraph &loop = g.ms_loop;
    const bool reuse = use_graph && loop.matches(&key, sizeof(key));
    if (use_graph) {
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
    HYT_CUDA(cudaMemcpyAsync(d_args, &a, sizeof(a), cudaMemcpyHostToDevice, s));
    HYT_CUDA(cudaMemcpyAsync(hdr, &h0, sizeof(h0), cudaMemcpyHostToDevice, s));
    ms_init_kernel<<<grid_for(V * kML, 256, 148 * 8), 256, 0, s>>>(d_args);
    ms_sources_kernel<<<1, 32, 0, s>>>(d_args);
    HYT_CUDA(cudaGetLastError());
    uint32_t launches = 2;
    if (use_graph && !reuse) {
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
        auto add = [&](const void *f, dim3 gd, dim3 bd, unsigned smem) {
            cudaKernelNodeParams kp = {};
            kp.func = const_cast<void *>(f);
            kp.gridDim = gd;
            kp.blockDim = bd;
            kp.sharedMemBytes = smem;
            kp.kernelParams = kargs;
            HYT_CUDA(cudaGraphAddKernelNode(&node, body, prev ? &prev : nullptr, prev ? 1 : 0, &kp));
            prev = node;
        };
        add(reinterpret_cast<void *>(ms_expand_kernel<WK, kB>), dim3(grid), dim3(kMSThreads), 0);
        add(reinterpret_cast<void *>(ms_hub_kernel<WK, kB>), dim3(grid), dim3(kMSThreads), 0);
        if (a.pull_div) {
            add(reinterpret_cast<void *>(ms_pull_kernel<WK, kB>), dim3(pgrid), dim3(kMPThreads), pull_smem);
            add(reinterpret_cast<void *>(ms_round_close_kernel), dim3(1), dim3(1), 0);
        } else {
            add(reinterpret_cast<void *>(ms_round_end_kernel), dim3(1), dim3(1), 0);
        }
        HYT_CUDA(cudaGraphInstantiate(&loop.exec, loop.graph, 0));
        loop.set_key(&key, sizeof(key));
    }
    if (use_graph) {
        HYT_CUDA(cudaGraphLaunch(loop.exec, s));
    } else {
        for (uint32_t r = 0; r < max_rounds; ++r) {
            ms_expand_kernel<WK, kB><<<grid, kMSThreads, 0, s>>>(d_args);
            ms_hub_kernel<WK, kB><<<grid, kMSThreads, 0, s>>>(d_args);
            if (a.pull_div) {
                ms_pull_kernel<WK, kB><<<pgrid, kMPThreads, pull_smem, s>>>(d_args);
                ms_round_close_kernel<<<1, 1, 0, s>>>(d_args);
            } else {
                ms_round_end_kernel<<<1, 1, 0, s>>>(d_args);
            }
            HYT_CUDA(cudaGetLastError());
            launches += a.pull_div ? 4 : 3;
            uint32_t done = 0;
            HYT_CUDA(cudaMemcpyAsync(&done, &hdr->done, sizeof(done), cudaMemcpyDeviceToHost, s));
            HYT_CUDA(cudaStreamSynchronize(s));
            if (done) break;
        }
    }
    MSHeader h{};
    HYT_CUDA(cudaMemcpyAsync(&h, hdr, sizeof(h), cudaMemcpyDeviceToHost, s));
    total.stop(s);
    const double total_ms = total.ms();
    if (use_graph) launches += (a.pull_div ? 4 : 3) * h.round;
    if (out) {
        if (is_device_pointer(out)) {
            ms_emit_kernel<<<grid_for(V, 256), 256, 0, s>>>(g.ms_dist.get(), g.inv.get(), V, k, a.inf, unreached, out);
            HYT_CUDA(cudaGetLastError());
        } else {
            Scratch<uint32_t> tmp(V * k, s);
            ms_emit_kernel<<<grid_for(V, 256), 256, 0, s>>>(g.ms_dist.get(), g.inv.get(), V, k, a.inf, unreached, tmp.get());
            HYT_CUDA(cudaGetLastError());
            copy_from_device(out, tmp.get(), V * k * sizeof(uint32_t), s);
        }
    }
    HYT_CUDA(cudaStreamSynchronize(s));
    if (stats) {
        stats->iterations = h.round;
        stats->converged = h.converged;
        stats->device_ms = total_ms;
        stats->total_launches = launches;
        stats->edges_processed = h.relaxations;
        stats->vertices_processed = h.frontier_total;
        // per frontier vertex: 8 B offset pair (read twice) + 32 B label row
        // + 4 B queue entry; per relaxed edge: 4 B column + 4 B weight + a
        // 32 B label row
        stats->algorithmic_bytes = 52ull * h.frontier_total + 40ull * h.relaxations;
    }
}

}  // namespace

void sssp_multi(GraphImpl &g, const uint32_t *sources, uint32_t k, uint32_t max_rounds, uint32_t flags,
                cudaStream_t s, uint32_t *out, hyt_run_stats *stats) {
    if (!(g.flags & HYT_GRAPH_PUSH)) fail(HYT_E_INVALID, "graph was created without HYT_GRAPH_PUSH");
    if (!sources) fail(HYT_E_INVALID, "sources is NULL");
    if (k == 0 || k > kML) fail(HYT_E_INVALID, "hyt_sssp_multi takes 1 to 8 sources");
    for (uint32_t l = 0; l < k; ++l)
        if (sources[l] >= g.V) fail(HYT_E_INVALID, "SSSP source vertex is out of range");
    if (!g.weights_ok) fail(HYT_E_INVALID, "SSSP requires finite non-negative edge weights");
    const uint64_t cap = std::min<uint64_t>(4 * g.V + 1024, 0x7FFFFFFFull);
    const uint32_t rounds = max_rounds ? max_rounds : static_cast<uint32_t>(cap);
    // bounded labels: packed words say so for u32 weights; unweighted paths
    // have at most V - 1 edges
    const uint32_t max_w = g.weight_kind == HYT_WEIGHTS_NONE ? 1u : g.weight_range.high;
    const bool bounded = g.weight_kind == HYT_WEIGHTS_NONE ? g.V < HYT_DIST_INF_U32 : g.in_pack_bits > 0;
    switch (g.weight_kind) {
        case HYT_WEIGHTS_NONE:
            if (bounded)
                ms_solve<HYT_WEIGHTS_NONE, true>(g, sources, k, rounds, flags, s, max_w, out, stats);
            else
                ms_solve<HYT_WEIGHTS_NONE, false>(g, sources, k, rounds, flags, s, max_w, out, stats);
            break;
        case HYT_WEIGHTS_U32:
            if (bounded)
                ms_solve<HYT_WEIGHTS_U32, true>(g, sources, k, rounds, flags, s, max_w, out, stats);
            else
                ms_solve<HYT_WEIGHTS_U32, false>(g, sources, k, rounds, flags, s, max_w, out, stats);
            break;
        case HYT_WEIGHTS_F32: ms_solve<HYT_WEIGHTS_F32, false>(g, sources, k, rounds, flags, s, max_w, out, stats); break;
        default: fail(HYT_E_INTERNAL, "unknown weight kind");
    }
}

}  // namespace hyt
