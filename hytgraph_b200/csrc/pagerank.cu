// PageRank and personalized PageRank: synchronous (Jacobi) pull over the CSC.
//
// Semantics follow the reference CPU solver (src/algorithms/pagerank.cpp:
// 89-163): x_0 = 1/n; each step
//     x'[v] = (1-d)/n + d * dangling / n + d * sum_{u->v} x[u] / deg(u)
// with dangling = sum of x over out-degree-0 vertices, residual = L1 change,
// stop when residual <= tolerance or after max_iterations.  Per-edge
// contributions x[u]/deg(u) are formed once per vertex in the producing
// step (the reference divides per edge, same float quotient).  In-row sums
// are compensated (TwoSum/Kahan) in FP32; residual and dangling mass are
// reduced in FP64.
//
// The whole solve is one cooperative kernel (pr_solve_kernel: 1024 threads, one
// CTA per SM, a grid barrier between the passes); out-of-HBM solves and solves
// launched kernel by kernel run pr_iterate_kernel over a range of tasks.  The
// work list is the graph's pull tasks, assigned to warps round-robin
// (warp w takes tasks w, w + W, ..., the last ones on demand):
//   chunk tasks  -- 1024- to 4096-edge slices of rows with in-degree >=
//                   tile_cost; each warp writes a compensated partial, the
//                   last arriving warp of a row merges the partials in chunk
//                   order;
//   tile tasks   -- merge-path tiles of consecutive shorter rows (512 or
//                   1024 units), 32 rows at a time: groups of 1 to 8 lanes,
//                   or the whole warp, gather a row's contributions and sum
//                   them in registers (tile_task).
//
// What bounds it: random 4-byte gathers cost one 32-byte L2 sector each, and
// an SM takes at most 1.02 sectors per clock (measured on a 64 MB table), but
// only with L1 to hold the outstanding misses: 0.85 per clock beside 132 KB of
// shared memory, 0.60 beside 164 KB, 0.28 beside 196 KB.  So nothing but the
// hot-source table lives in shared memory.  The former layout staged every
// tile's contributions in 4 KB per warp (132 KB per CTA) and ran an iteration
// of R-MAT scale 24 (263 M edges, 8192 hot sources) in 1.16 ms; sums in
// registers take 1.02 ms.
//
// Results are deterministic: every row sum has a fixed association order,
// and the FP64 residual and dangling mass are summed in a fixed slot order
// (PRSlots), independent of the grid size and of warp arrival order: each
// task stores its slot, then the reduction sums the slots and evaluates the
// stop rule.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "graph.cuh"
#include "grid_sync.cuh"
#include "hybrid.cuh"
#include "pagerank_core.cuh"
#include "solvers.cuh"

namespace hyt {
namespace {

using namespace prc;

// Slot of long row i and of tile k in the fixed-order reduction.
__device__ __forceinline__ uint32_t long_slot(uint32_t i) { return i; }
__device__ __forceinline__ uint32_t tile_slot(const PRArgs &a, uint64_t k) {
    return a.red.num_slots - static_cast<uint32_t>(a.num_tiles) + static_cast<uint32_t>(k);
}

// Hot-source contributions of this iteration, loaded once per CTA.
__device__ __forceinline__ void load_hot(const PRArgs &a, const PRBuffers &b, float *s_hot) {
    const uint32_t nt = blockDim.x;
    if (threadIdx.x == 0) s_hot[a.num_hot] = 0.0f;  // "no edge"
    for (uint32_t i0 = 0; i0 < a.num_hot; i0 += 8 * nt) {
        uint32_t hv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t i = i0 + k * nt + threadIdx.x;
            hv[k] = (i < a.num_hot) ? a.hot_vertex[i] : 0u;
        }
        float hc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) hc[k] = b.ccur[hv[k]];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t i = i0 + k * nt + threadIdx.x;
            if (i < a.num_hot) s_hot[i] = hc[k];
        }
    }
}

// One launch processes chunk tasks [chunk_begin, chunk_end) and tiles
// [tile_begin, tile_end); in_src is the base of the source ids, addressed by
// global edge index (a device array, a staging slot offset by its first
// edge, or mapped host memory).  An iteration may span several launches;
// pr_reduce_kernel closes it after the last one.
struct PRRange {
    const uint32_t *in_src;
    uint64_t chunk_begin, chunk_end, tile_begin, tile_end;
    const uint4 *tasks;  // the graph's task descriptors (whole-graph launches; NULL: no prefetch)
    union {
        uint64_t dealt;      // dealt_tasks (whole-graph launches)
        const uint2 *whole;  // launches over pieces: rows of the tile that tile k is a part of
    };
};

// The tasks of one iteration, over the whole grid.  a: the solve's arguments
// as kernel parameters (the constant bank: no registers held across the
// tasks).
// cursor (whole-graph launches): the first rg.dealt tasks are dealt to the
// warps in turn, the others taken one by one.
// kPieces: a launch over out-of-HBM pieces, whose tasks have no descriptors and
// whose tiles are parts of tiles.
template <bool kPieces>
__device__ __forceinline__ void run_tasks(const PRArgs &a, const PRRange &rg, const PRState &ps, const PRBuffers &b,
                                          double2 *slots, float *s_hot, uint32_t *cursor) {
    const uint64_t n_chunks = rg.chunk_end - rg.chunk_begin;
    const uint64_t total_tasks = n_chunks + (rg.tile_end - rg.tile_begin);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    load_hot(a, b, s_hot);
    __syncthreads();
    const uint64_t nwarps = uint64_t(gridDim.x) * (kPRThreads / 32);
    uint64_t task = uint64_t(blockIdx.x) * (kPRThreads / 32) + warp;
    const uint64_t dealt = cursor ? max(rg.dealt, min(total_tasks, nwarps)) : total_tasks;
    // whole-graph launches read a dealt task's descriptor while the task
    // before it runs (one 16-byte load in place of a chain of table reads)
    uint4 d = (rg.tasks && task < total_tasks) ? rg.tasks[task] : make_uint4(0, 0, 0, 0);
    while (task < total_tasks) {
        double res = 0.0, dang = 0.0;
        uint64_t next = task + nwarps;
        uint32_t ticket = 0;
        const bool ask = cursor && next >= dealt;
        if (ask && lane == 0) ticket = atomicAdd(cursor, 1u);
        uint4 nd = (rg.tasks && next < dealt) ? rg.tasks[next] : make_uint4(0, 0, 0, 0);
        const uint4 *pf = (rg.tasks && !ask) ? &nd : nullptr;
        if (task < n_chunks) {
            const TaskSpan t = rg.tasks ? task_span(d) : chunk_span(a, rg.chunk_begin + task);
            const uint32_t row = chunk_task<true>(a, ps, b, rg.in_src, s_hot, t, lane, res, dang, pf);
            if (row != ~0u) slot_store(slots, long_slot(row), dev::warp_sum(res), dev::warp_sum(dang), lane);
        } else {
            const uint64_t k = rg.tile_begin + (task - n_chunks);
            const TaskSpan t = rg.tasks ? task_span(d) : tile_span(a, k);
            tile_task<true, kPieces>(a, ps, b, rg.in_src, s_hot, t, lane, res, dang, pf,
                                     kPieces ? rg.whole[k] : make_uint2(0, 0));
            slot_store(slots, tile_slot(a, k), dev::warp_sum(res), dev::warp_sum(dang), lane);
        }
        if (ask) {
            next = dealt + __shfl_sync(0xffffffffu, ticket, 0);
            if (rg.tasks && next < total_tasks) nd = rg.tasks[next];
        }
        task = next;
        d = nd;
    }
}

// One iteration (or a part of one: out-of-HBM partitions); the scalars of
// this solve are in *args.
template <bool kPieces>
__global__ void __launch_bounds__(kPRThreads, 1) pr_iterate_kernel(const PRArgs *__restrict__ args,
                                                                   const __grid_constant__ PRArgs a,
                                                                   const __grid_constant__ PRRange rg) {
    extern __shared__ __align__(16) float s_dyn[];
    const uint32_t it = *(volatile uint32_t *)&a.hdr->iter;
    if (*(volatile uint32_t *)&a.hdr->done) return;
    run_tasks<kPieces>(a, rg, make_state(*args, a.dangling[it]), buffers(a, it), a.red.slot, s_dyn, nullptr);
}

// (residual, dangling) of slot group g: thread t of 256 takes slots t, t +
// 256, ..., then a fixed tree.  Called by 256 consecutive threads (8 warps, of
// which warp `w`); s_part holds 8 entries of theirs; the result is in lane 0
// of their first warp after the caller's barrier and fold_group.
constexpr int kReduceThreads = 256;

__device__ __forceinline__ double2 group_part(const PRSlots &R, const double2 *slots, uint32_t g, uint32_t t) {
    const uint32_t b = g * kSlotGroup, n = min(kSlotGroup, R.num_slots - b);
    double r = 0.0, d = 0.0;
    for (uint32_t i = t; i < n; i += kReduceThreads) {
        const double2 x = __ldcg(slots + b + i);
        r += x.x;
        d += x.y;
    }
    return make_double2(dev::warp_sum(r), dev::warp_sum(d));
}

__device__ __forceinline__ double2 fold_group(const double2 *s_part, int lane) {
    const double2 v = lane < kReduceThreads / 32 ? s_part[lane] : make_double2(0.0, 0.0);
    return make_double2(dev::warp_sum(v.x), dev::warp_sum(v.y));
}

// The whole solve in one cooperative launch: iterations separated by grid
// barriers in place of two kernel launches and a conditional-graph step each
// (on 65 K edges those cost more than the work; the graph was also built and
// instantiated for every solve): 523 -> 235 us a call on 4099 vertices and 65 K
// edges, 19.7 -> 19.4 ms on R-MAT scale 24.  Every CTA takes the stop decision by itself
// from the same sums.  Up to kOwnGroups slot groups are summed by every CTA
// (one barrier an iteration); more are shared out, with a second barrier.
// Slots alternate between two halves, so an iteration's slots are not
// overwritten before every CTA has passed the next barrier.  The sums'
// association is that of pr_reduce_kernel.
constexpr uint32_t kOwnGroups = kPRThreads / kReduceThreads;

__global__ void __launch_bounds__(kPRThreads, 1) pr_solve_kernel(const __grid_constant__ PRArgs a,
                                                                 const __grid_constant__ PRRange rg) {
    extern __shared__ __align__(16) float s_dyn[];
    __shared__ double2 s_part[kPRThreads / 32];
    __shared__ double2 s_group[kOwnGroups];
    __shared__ double2 s_total;
    const PRSlots &R = a.red;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t sub = threadIdx.x / kReduceThreads, t = threadIdx.x % kReduceThreads;
    constexpr int kSubWarps = kReduceThreads / 32;
    uint32_t barriers = 0;
    double dangling = a.dangling[0];
    bool ok = true;
    for (uint32_t it = 0; ok; ++it) {
        double2 *slots = R.slot + ((it & 1) ? R.num_slots : 0);
        // three cursors take turns: this one was cleared two iterations ago
        if (blockIdx.x == 0 && threadIdx.x == 0) R.blocks_done[1 + (it + 2) % 3] = 0;
        run_tasks<false>(a, rg, make_state(a, dangling), buffers(a, it), slots, s_dyn, R.blocks_done + 1 + it % 3);
        ok = dev::grid_sync(R.blocks_done, barriers);
        if (!ok) break;
        const bool own = R.num_groups <= kOwnGroups;
        const uint32_t first = own ? sub : blockIdx.x * kOwnGroups + sub;
        const uint32_t step = own ? kOwnGroups : gridDim.x * kOwnGroups;
        const uint32_t rounds = (R.num_groups + step - 1) / step;
        for (uint32_t k = 0; k < rounds; ++k) {
            const uint32_t g = first + k * step;
            double2 p = make_double2(0.0, 0.0);
            if (g < R.num_groups) p = group_part(R, slots, g, t);
            if (lane == 0) s_part[warp] = p;
            __syncthreads();
            if (warp % kSubWarps == 0 && g < R.num_groups) {
                const double2 v = fold_group(s_part + sub * kSubWarps, lane);
                if (lane == 0) {
                    if (own)
                        s_group[sub] = v;
                    else
                        R.group_sum[g] = v;
                }
            }
            __syncthreads();
        }
        if (!own) {
            ok = dev::grid_sync(R.blocks_done, barriers);
            if (!ok) break;
        }
        if (warp == 0) {
            double r = 0.0, d = 0.0;
            for (uint32_t g = lane; g < R.num_groups; g += 32) {
                const double2 x = own ? s_group[g] : __ldcg(R.group_sum + g);
                r += x.x;
                d += x.y;
            }
            r = dev::warp_sum(r);
            d = dev::warp_sum(d);
            if (lane == 0) s_total = make_double2(r, d);
        }
        __syncthreads();
        const double2 total = s_total;
        dangling = total.y;
        const bool done = total.x <= static_cast<double>(a.tolerance) || it + 1 >= a.max_iter;
        if (blockIdx.x == 0 && threadIdx.x == 0) close_iteration(a, it, total.x, total.y);
        if (done) return;
        __syncthreads();  // s_total and the hot table are rewritten
    }
    if (threadIdx.x == 0) atomicExch(&a.hdr->error, 1u);
}

// Closes an iteration: block b sums slot groups b, b + grid, ... (thread t
// takes slots t, t + 256, ... of the group, then a fixed block tree); the
// last block to finish sums the group sums in group order, then applies
// the stop rule.
__global__ void __launch_bounds__(kReduceThreads) pr_reduce_kernel(const PRArgs *__restrict__ args) {
    __shared__ double s_red[32];
    __shared__ uint32_t s_last;
    const PRArgs a = *args;
    if (*(volatile uint32_t *)&a.hdr->done) return;
    const uint32_t it = *(volatile uint32_t *)&a.hdr->iter;
    const PRSlots &R = a.red;
    for (uint32_t g = blockIdx.x; g < R.num_groups; g += gridDim.x) {
        const uint32_t b = g * kSlotGroup, n = min(kSlotGroup, R.num_slots - b);
        double r = 0.0, d = 0.0;
        for (uint32_t i = threadIdx.x; i < n; i += kReduceThreads) {
            const double2 x = __ldcg(R.slot + b + i);
            r += x.x;
            d += x.y;
        }
        r = dev::block_sum(r, s_red);
        __syncthreads();
        d = dev::block_sum(d, s_red);
        if (threadIdx.x == 0) R.group_sum[g] = make_double2(r, d);
        __syncthreads();
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(R.blocks_done, 1u) + 1u == (it + 1) * gridDim.x) ? 1u : 0u;
    __syncthreads();
    if (!s_last || threadIdx.x >= 32) return;
    __threadfence();
    double r = 0.0, d = 0.0;
    for (uint32_t g = threadIdx.x; g < R.num_groups; g += 32) {
        const double2 x = __ldcg(R.group_sum + g);
        r += x.x;
        d += x.y;
    }
    r = dev::warp_sum(r);
    d = dev::warp_sum(d);
    if (threadIdx.x == 0) close_iteration(a, it, r, d);
}

// Initial ranks and contributions; the initial dangling mass is summed in a
// fixed order: per kInitChunk-vertex chunk (a fixed thread mapping and block
// tree), then the chunk partials in chunk order by the last block.
constexpr uint32_t kInitChunk = 4096;
constexpr int kInitThreads = 256;

__global__ void __launch_bounds__(kInitThreads) pr_init_kernel(const __grid_constant__ PRArgs a, double *part,
                                                               uint32_t *count) {
    __shared__ double s_red[32];
    __shared__ uint32_t s_last;
    const uint32_t V = a.V;
    const uint32_t nchunks = (V + kInitChunk - 1) / kInitChunk;
    const float r0_uniform = __fdiv_rn(1.0f, static_cast<float>(V));
    for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        double dang = 0.0;
        const uint32_t end = min(V, (c + 1) * kInitChunk);
        for (uint32_t v = c * kInitChunk + threadIdx.x; v < end; v += kInitThreads) {
            const float r0 = a.personalized ? (v == a.source ? 1.0f : 0.0f) : r0_uniform;
            a.rank[0][v] = r0;
            const uint32_t od = a.out_deg[v];
            a.contrib[0][v] = od ? __fdiv_rn(r0, static_cast<float>(od)) : 0.0f;
            if (od == 0) dang += r0;
        }
        const double bsum = dev::block_sum(dang, s_red);
        if (threadIdx.x == 0) part[c] = bsum;
        __syncthreads();
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(count, 1u) + 1u == gridDim.x) ? 1u : 0u;
    __syncthreads();
    if (!s_last || threadIdx.x >= 32) return;
    __threadfence();
    double d = 0.0;
    for (uint32_t i = threadIdx.x; i < nchunks; i += 32) d += __ldcg(part + i);
    d = dev::warp_sum(d);
    if (threadIdx.x == 0) a.dangling[0] = d;
}

// Persistent grid of the iteration kernels: one CTA per SM, or HYT_PR_GRID
// CTAs (results do not depend on it).
int pr_occupancy_grid() {
    static int grid = 0;
    if (grid == 0) {
        int per_sm = 0;
        HYT_CUDA(cudaFuncSetAttribute(pr_iterate_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kPRSmemMax)));
        HYT_CUDA(cudaFuncSetAttribute(pr_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kPRSmemMax - 4096)));
        HYT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pr_iterate_kernel<false>, kPRThreads, kPRSmemMax));
        grid = sm_count() * std::max(per_sm, 1);
        if (const char *e = std::getenv("HYT_PR_GRID")) {
            const long v = std::strtol(e, nullptr, 10);
            if (v > 0 && v <= 65535) grid = static_cast<int>(v);
        }
    }
    return grid;
}

}  // namespace

// Shared by PageRank and personalized PageRank.
// Workspaces, device state layout and kernel arguments of one solve.
struct PRSolveState {
    PRArgs a;
    PRArgs *d_args;
    PRHeader *hdr;
    size_t zero_bytes;
    double *init_part;
    uint32_t *init_count;
};

// pr_state layout: args | header | residual[max_iter] | dangling[max_iter+1]
// | init partials | init counter | reduce-blocks counter, 3 task cursors |
// (16-byte aligned)
// group sums | slots.  Everything from the header through the counters is
// cleared at the start of a solve.
static PRSolveState pr_prepare(GraphImpl &g, bool personalized, uint32_t source, float damping, float tolerance,
                               uint32_t max_iter) {
    const uint64_t V = g.V;
    // Workspaces (grown on demand, kept in the handle).
    for (int i = 0; i < 2; ++i) {
        if (g.rank[i].count < V) g.rank[i].allocate(V);
        if (g.contrib[i].count < V) g.contrib[i].allocate(V);
    }
    if (g.partial.count < 2 * std::max<uint64_t>(g.num_chunks, 1)) g.partial.allocate(2 * std::max<uint64_t>(g.num_chunks, 1));
    if (g.ticket.count < std::max<uint64_t>(g.num_long, 1)) g.ticket.allocate(std::max<uint64_t>(g.num_long, 1));
    const uint64_t num_slots = g.num_long + g.num_tiles;
    if (num_slots > 0xFFFFFFFFull) fail(HYT_E_UNSUPPORTED, "PageRank: too many pull tasks for one graph");
    const uint64_t num_groups = (num_slots + kSlotGroup - 1) / kSlotGroup;
    const uint64_t init_chunks = (V + kInitChunk - 1) / kInitChunk;
    auto up16 = [](size_t x) { return (x + 15) & ~size_t(15); };  // double2 needs 16-byte alignment
    const size_t args_bytes = (sizeof(PRArgs) + 255) & ~size_t(255);
    const size_t head = sizeof(PRHeader) + size_t(max_iter) * sizeof(double) + size_t(max_iter + 1) * sizeof(double) +
                        size_t(init_chunks) * sizeof(double) + 5 * sizeof(uint32_t);
    const size_t sb = args_bytes + up16(head) + size_t(num_groups + 2 * num_slots) * sizeof(double2) + 64;
    if (g.pr_state.count < sb) g.pr_state.allocate(sb);

    unsigned char *base = g.pr_state.get();
    PRArgs *d_args = reinterpret_cast<PRArgs *>(base);
    unsigned char *p = base + args_bytes;
    PRHeader *hdr = reinterpret_cast<PRHeader *>(p);
    p += sizeof(PRHeader);
    double *residual = reinterpret_cast<double *>(p);
    p += size_t(max_iter) * sizeof(double);
    double *dangling = reinterpret_cast<double *>(p);
    p += size_t(max_iter + 1) * sizeof(double);
    double *init_part = reinterpret_cast<double *>(p);
    p += size_t(init_chunks) * sizeof(double);
    uint32_t *init_count = reinterpret_cast<uint32_t *>(p);
    p += sizeof(uint32_t);
    uint32_t *blocks_done = reinterpret_cast<uint32_t *>(p);
    p += 4 * sizeof(uint32_t);
    const size_t zero_bytes = static_cast<size_t>(p - reinterpret_cast<unsigned char *>(hdr));
    p = base + args_bytes + up16(head);
    double2 *group_sum = reinterpret_cast<double2 *>(p);
    p += size_t(num_groups) * sizeof(double2);
    double2 *slots = reinterpret_cast<double2 *>(p);
    if (reinterpret_cast<uintptr_t>(base) % 256 || reinterpret_cast<uintptr_t>(group_sum) % 16 ||
        reinterpret_cast<uintptr_t>(slots) % 16 || reinterpret_cast<uintptr_t>(residual) % 8)
        fail(HYT_E_INTERNAL, "PageRank state layout is misaligned");

    PRArgs a{};
    a.in_off = g.in_offsets.get();
    a.in_src = g.in_sources.get();
    a.out_deg = g.out_degree.get();
    a.tile_start = g.tile_start.get();
    a.long_rows = g.long_rows.get();
    a.chunk_tasks = g.chunk_tasks.get();
    a.hot_vertex = g.hot_vertex.get();
    a.num_hot = g.num_hot;
    a.tile_cost = g.tile_cost;
    a.chunk_edges = g.chunk_edges;
    for (int i = 0; i < 2; ++i) {
        a.rank[i] = g.rank[i].get();
        a.contrib[i] = g.contrib[i].get();
    }
    a.partial = reinterpret_cast<float2 *>(g.partial.get());
    a.ticket = g.ticket.get();
    a.hdr = hdr;
    a.residual = residual;
    a.dangling = dangling;
    a.num_tiles = g.num_tiles;
    a.num_chunks = static_cast<uint32_t>(g.num_chunks);
    a.V = static_cast<uint32_t>(V);
    a.damping = damping;
    a.base = personalized ? 0.0f : (1.0f - damping) / static_cast<float>(V);
    a.tolerance = tolerance;
    a.max_iter = max_iter;
    a.source = source;
    a.personalized = personalized ? 1u : 0u;
    a.red = PRSlots{slots, group_sum, blocks_done, static_cast<uint32_t>(num_slots),
                    static_cast<uint32_t>(num_groups)};
    a.tasks = g.pull_tasks.get();

    return PRSolveState{a, d_args, hdr, zero_bytes, init_part, init_count};
}

static void pr_check_header(const PRHeader &h) {
    if (h.error) fail(HYT_E_TIMEOUT, "PageRank: a bounded wait at a grid barrier ran out");
    if (h.iter == 0) fail(HYT_E_INTERNAL, "PageRank made no progress");
}

// Grid of the per-iteration reduce kernel (fixed for a solve).
static unsigned pr_reduce_grid(const PRArgs &a) {
    return static_cast<unsigned>(std::max<uint32_t>(1u, std::min<uint32_t>(a.red.num_groups, 148u * 4)));
}

static void pr_init(const PRSolveState &st, uint64_t V, cudaStream_t s) {
    const unsigned blocks = static_cast<unsigned>(std::min<uint64_t>((V + kInitChunk - 1) / kInitChunk, 148ull * 8));
    pr_init_kernel<<<blocks, kInitThreads, 0, s>>>(st.a, st.init_part, st.init_count);
    HYT_CUDA(cudaGetLastError());
}

static void pr_solve(GraphImpl &g, bool personalized, uint32_t source, float damping, float tolerance,
                     uint32_t max_iter, uint32_t flags, cudaStream_t s, float *ranks_out, hyt_run_stats *stats) {
    if (!(g.flags & HYT_GRAPH_PULL)) fail(HYT_E_INVALID, "graph was created without HYT_GRAPH_PULL");
    const uint64_t V = g.V;
    PRSolveState st0 = pr_prepare(g, personalized, source, damping, tolerance, max_iter);
    PRArgs &a = st0.a;
    PRArgs *d_args = st0.d_args;
    PRHeader *hdr = st0.hdr;
    // one persistent launch, or (profiling, launch-by-launch runs) a host loop
    const bool persistent = !(flags & HYT_RUN_NO_GRAPH) && !(flags & HYT_RUN_PROFILE);
    const int grid = pr_occupancy_grid();
    const unsigned smem = static_cast<unsigned>(pr_hot_bytes(g.num_hot));
    PRRange full{g.in_sources.get(), 0, g.num_chunks, 0, g.num_tiles, g.pull_tasks.get(), {dealt_tasks(g)}};

    EventTimer total;
    total.start(s);
    HYT_CUDA(cudaMemsetAsync(hdr, 0, st0.zero_bytes, s));
    HYT_CUDA(cudaMemsetAsync(g.ticket.get(), 0, g.ticket.bytes(), s));

    uint32_t launches = 0, hot_launches = 0;
    double kernel_ms = 0.0;
    pr_init(st0, V, s);
    ++launches;

    if (persistent) {
        // every CTA must be resident; no more of them than have tasks
        const uint64_t tasks = g.num_chunks + g.num_tiles;
        const unsigned ctas = static_cast<unsigned>(
            std::min<uint64_t>({static_cast<uint64_t>(grid), static_cast<uint64_t>(sm_count()),
                                std::max<uint64_t>(1, (tasks + kPRThreads / 32 - 1) / (kPRThreads / 32))}));
        void *kargs[] = {&a, &full};
        HYT_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(pr_solve_kernel), dim3(ctas), dim3(kPRThreads),
                                             kargs, smem, s));
        ++launches;
    } else {
        HYT_CUDA(cudaMemcpyAsync(d_args, &a, sizeof(PRArgs), cudaMemcpyHostToDevice, s));
        EventTimer kt;
        for (uint32_t i = 0; i < max_iter; ++i) {
            if (flags & HYT_RUN_PROFILE) kt.start(s);
            pr_iterate_kernel<false><<<grid, kPRThreads, smem, s>>>(d_args, a, full);
            pr_reduce_kernel<<<pr_reduce_grid(a), kReduceThreads, 0, s>>>(d_args);
            HYT_CUDA(cudaGetLastError());
            launches += 2;
            if (flags & HYT_RUN_PROFILE) {
                kt.stop(s);
                const double ms = kt.ms();
                uint32_t done = 0;
                HYT_CUDA(cudaMemcpyAsync(&done, &hdr->done, sizeof(done), cudaMemcpyDeviceToHost, s));
                HYT_CUDA(cudaStreamSynchronize(s));
                kernel_ms += ms;
                ++hot_launches;
                if (done) break;
            } else if ((i & 3) == 3) {
                uint32_t done = 0;
                HYT_CUDA(cudaMemcpyAsync(&done, &hdr->done, sizeof(done), cudaMemcpyDeviceToHost, s));
                HYT_CUDA(cudaStreamSynchronize(s));
                if (done) break;
            }
        }
    }
    PRHeader local{};
    PRHeader *hp = g.host_scratch.ptr ? reinterpret_cast<PRHeader *>(g.host_scratch.ptr) : &local;
    HYT_CUDA(cudaMemcpyAsync(hp, hdr, sizeof(PRHeader), cudaMemcpyDeviceToHost, s));
    total.stop(s);
    const double total_ms = total.ms();
    const PRHeader h = *hp;
    pr_check_header(h);
    if (ranks_out) graph_emit(g, ranks_out, g.rank[h.iter & 1].get(), s);

    if (stats) {
        stats->iterations = h.iter;
        stats->converged = h.converged;
        stats->residual = h.last_residual;
        stats->device_ms = total_ms;
        stats->kernel_ms = kernel_ms;
        stats->kernel_launches = hot_launches;
        stats->total_launches = launches;
        stats->edges_processed = uint64_t(h.iter) * g.E;
        stats->vertices_processed = uint64_t(h.iter) * V;
        // 4 B source id + 4 B gathered contribution per edge; 8 B CSC offset
        // + 4 B rank read + 4 B rank write + 4 B contribution write per vertex.
        stats->algorithmic_bytes = uint64_t(h.iter) * (8ull * g.E + 20ull * V);
    }
}

void pagerank_run(GraphImpl &g, const hyt_pagerank_params &p, float *ranks_out, hyt_run_stats *stats) {
    if (!(p.damping >= 0.0f && p.damping < 1.0f)) fail(HYT_E_INVALID, "PageRank damping_factor must be in [0, 1)");
    if (!(p.tolerance > 0.0f) || !std::isfinite(p.tolerance))
        fail(HYT_E_INVALID, "PageRank tolerance must be finite and positive");
    if (p.max_iterations == 0) fail(HYT_E_INVALID, "PageRank max_iterations must be greater than zero");
    cudaStream_t s = p.stream ? static_cast<cudaStream_t>(p.stream) : g.stream;
    pr_solve(g, false, 0, p.damping, p.tolerance, p.max_iterations, p.flags, s, ranks_out, stats);
}

void ppr_run(GraphImpl &g, const hyt_ppr_params &p, float *ranks_out, hyt_run_stats *stats) {
    if (!(p.restart > 0.0f && p.restart <= 1.0f)) fail(HYT_E_INVALID, "personalized PageRank restart must be in (0, 1]");
    if (!(p.tolerance > 0.0f) || !std::isfinite(p.tolerance))
        fail(HYT_E_INVALID, "personalized PageRank tolerance must be finite and positive");
    if (p.max_iterations == 0) fail(HYT_E_INVALID, "personalized PageRank max_iterations must be greater than zero");
    if (p.source >= g.V) fail(HYT_E_INVALID, "personalized PageRank source vertex is out of range");
    cudaStream_t s = p.stream ? static_cast<cudaStream_t>(p.stream) : g.stream;
    pr_solve(g, true, graph_vertex(g, p.source, s), 1.0f - p.restart, p.tolerance, p.max_iterations, p.flags, s,
             ranks_out, stats);
}

void pagerank_partitioned(GraphImpl &g, PullSource &src, bool personalized, uint32_t source, float damping,
                          float tolerance, uint32_t max_iter, cudaStream_t s, float *ranks_out, hyt_run_stats *stats) {
    const uint64_t V = g.V;
    PRSolveState st0 = pr_prepare(g, personalized, source, damping, tolerance, max_iter);
    const PRArgs &a = st0.a;
    const int grid = pr_occupancy_grid();
    const size_t smem = pr_hot_bytes(a.num_hot);

    EventTimer total;
    total.start(s);
    HYT_CUDA(cudaMemsetAsync(st0.hdr, 0, st0.zero_bytes, s));
    HYT_CUDA(cudaMemsetAsync(g.ticket.get(), 0, g.ticket.bytes(), s));
    HYT_CUDA(cudaMemcpyAsync(st0.d_args, &a, sizeof(PRArgs), cudaMemcpyHostToDevice, s));
    pr_init(st0, V, s);
    uint32_t launches = 1, hot = 0;
    PRHeader h{};
    for (uint32_t it = 0; it < max_iter; ++it) {
        src.begin_iteration(s);
        for (size_t p = 0; p < src.parts();) {
            // Pieces readable together, with consecutive tasks, share a launch: a
            // launch's time is that of its slowest task, not its size.  16 M
            // edges in 64 partitions, 32 MB on the device: 71 launches an
            // iteration -> 40, 16 iterations 31.9 -> 22.8 ms (shorter tasks
            // of long rows included).
            PullPart run = src.part(p);
            size_t last = p;
            while (src.joined(last)) {
                const PullPart nx = src.part(last + 1);
                if (nx.chunk_begin != run.chunk_end || nx.tile_begin != run.tile_end) break;
                run.chunk_end = nx.chunk_end;
                run.tile_end = nx.tile_end;
                ++last;
            }
            const bool any = run.chunk_begin != run.chunk_end || run.tile_begin != run.tile_end;
            const uint32_t *base = nullptr;
            for (size_t q = p; q <= last; ++q) base = src.acquire(q, s);
            if (any) {
                PRRange rg{base, run.chunk_begin, run.chunk_end, run.tile_begin, run.tile_end, nullptr, {0}};
                rg.whole = src.whole_tiles();
                pr_iterate_kernel<true><<<grid, kPRThreads, smem, s>>>(st0.d_args, a, rg);
                HYT_CUDA(cudaGetLastError());
                ++launches;
                ++hot;
            }
            for (size_t q = p; q <= last; ++q) src.release(q, s);
            p = last + 1;
        }
        pr_reduce_kernel<<<pr_reduce_grid(a), kReduceThreads, 0, s>>>(st0.d_args);
        HYT_CUDA(cudaGetLastError());
        ++launches;
        // the reduce kernel closed the iteration
        HYT_CUDA(cudaMemcpyAsync(&h, st0.hdr, sizeof(h), cudaMemcpyDeviceToHost, s));
        HYT_CUDA(cudaStreamSynchronize(s));
        if (h.error) break;
        if (h.iter != it + 1) fail(HYT_E_INTERNAL, "partitioned PageRank: an iteration left tasks unprocessed");
        if (h.done) break;
    }
    total.stop(s);
    const double total_ms = total.ms();
    pr_check_header(h);
    if (ranks_out) copy_from_device(ranks_out, g.rank[h.iter & 1].get(), V * sizeof(float), s);
    if (stats) {
        stats->iterations = h.iter;
        stats->converged = h.converged;
        stats->residual = h.last_residual;
        stats->device_ms = total_ms;
        stats->kernel_launches = hot;
        stats->total_launches = launches;
        stats->edges_processed = uint64_t(h.iter) * g.E;
        stats->vertices_processed = uint64_t(h.iter) * V;
        stats->algorithmic_bytes = uint64_t(h.iter) * (8ull * g.E + 20ull * V);
    }
}

}  // namespace hyt
