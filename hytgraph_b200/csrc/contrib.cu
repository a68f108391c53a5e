// Contribution-driven scheduling on the GPU: hyt_pagerank_contributions,
// hyt_sssp_contributions, hyt_contribution_schedule,
// hyt_partition_contributions.
//
// Contributions follow the reference's definitions
// (src/algorithms/pagerank.cpp:165-241, src/algorithms/sssp.cpp:236-290):
//   PageRank: |next(v) - current(v)| of one synchronous pull step,
//     next(v) = (1 - d)/n + d * dangling / n + d * sum_{u->v} current(u)/deg(u);
//     here the sums run in FP64 (each row in a fixed association over 1 to 8
//     lanes or a warp; dangling mass by per-block partials summed in a fixed
//     order), so the values are deterministic and agree with the reference's
//     FP32 to within its rounding;
//   SSSP: current - candidate when both are finite and the improvement
//     exceeds the tolerance, 1 when an unreachable vertex becomes
//     reachable, else 0 — the same FP32 operations, bit for bit.
// The schedule follows ContributionScheduler::schedule
// (src/scheduling/contribution_scheduler.cpp:23-121): items by descending
// contribution, ties by lower item index (deterministic tie-break; or input
// order otherwise), computed as stable radix sorts (item index where the items
// do not ascend already, then contribution), with the plan metrics (reordered, zero, redundant,
// log2(n) overhead).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cub/cub.cuh>

#include "common.cuh"
#include "graph.cuh"
#include "scratch.cuh"
#include "solvers.cuh"

namespace hyt {
namespace {

constexpr int kPartBlocks = 1024;

// x[u] = current(u) / deg(u) in FP64 (0 for a dangling vertex), and the
// per-block partial sums of the dangling ranks; clears the task cursor.
__global__ void source_shares_kernel(const uint32_t *__restrict__ deg, const float *__restrict__ rank, uint64_t V,
                                     double *__restrict__ x, double *__restrict__ partial, uint32_t *cursor) {
    __shared__ double warp_sum[8];
    if (blockIdx.x == 0 && threadIdx.x == 0) *cursor = 0;
    double acc = 0.0;
    for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < V; v += uint64_t(gridDim.x) * blockDim.x) {
        const uint32_t d = deg[v];
        const double r = rank[v];
        x[v] = d ? r / double(d) : 0.0;
        if (d == 0) acc += r;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) warp_sum[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += warp_sum[w];
        partial[blockIdx.x] = s;
    }
}

// In-edges of one task, addressed relative to its first edge.
struct InEdges {
    const uint32_t *src;    // source ids, hot ones tagged kHotTag | slot
    const uint32_t *s_hot;  // vertex ids of the hot slots
    const double *x;
};

// Sum of x over the edges b, b + kStep, ... below e, at most kN of them, all
// loaded before the first is added.
template <int kN, int kStep>
__device__ __forceinline__ double edges_sum(const InEdges &E, uint32_t b, uint32_t e, double acc) {
    uint32_t u[kN];
#pragma unroll
    for (int j = 0; j < kN; ++j) u[j] = (b + j * kStep < e) ? dev::ld_stream(E.src + b + j * kStep) : 0u;
#pragma unroll
    for (int j = 0; j < kN; ++j)
        if (u[j] & kHotTag) u[j] = E.s_hot[u[j] & ~kHotTag];
    double v[kN];
#pragma unroll
    for (int j = 0; j < kN; ++j) v[j] = (b + j * kStep < e) ? __ldg(E.x + u[j]) : 0.0;
#pragma unroll
    for (int j = 0; j < kN; ++j) acc += v[j];
    return acc;
}

// Sum over edges [b, e) by the whole warp; every lane returns it.
__device__ __forceinline__ double span_sum(const InEdges &E, uint32_t b, uint32_t e, int lane) {
    double acc = 0.0;
    for (uint32_t at = b; at < e; at += 256) {
        if (e - at <= 128)
            acc = edges_sum<4, 32>(E, at + lane, e, acc);
        else
            acc = edges_sum<8, 32>(E, at + lane, e, acc);
    }
    return dev::warp_sum(acc);
}

// Sums of the warp's 32 rows (lane l: edges [lo, hi)), kG lanes per row and
// 32 / kG rows a step; rows have at most kG * kN in-edges.
template <int kG, int kN>
__device__ __forceinline__ double group_sum(const InEdges &E, uint32_t lo, uint32_t hi, int lane) {
    constexpr int kRows = 32 / kG;
    double mine = 0.0;
    for (int step = 0; step < kG; ++step) {
        const int owner = step * kRows + lane / kG;
        const uint32_t b = __shfl_sync(0xffffffffu, lo, owner) + (lane % kG);
        const uint32_t e = __shfl_sync(0xffffffffu, hi, owner);
        double acc = edges_sum<kN, kG>(E, b, e, 0.0);
#pragma unroll
        for (int o = 1; o < kG; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        const double t = __shfl_sync(0xffffffffu, acc, (lane % kRows) * kG);
        if (lane / kRows == step) mine = t;
    }
    return mine;
}

// (1 - d)/n + d * dangling / n from the per-block dangling partials, summed
// by the block's first warp in a fixed order (lane l: partials l, l + 32,
// ...; then a shuffle tree), so no thread waits on one load per partial.
// Called by the first 32 threads; the result is in all of them.
__device__ __forceinline__ double base_share(const double *__restrict__ partial, int parts, uint64_t V, double d,
                                             int lane) {
    double dm = 0.0;
    for (int i = lane; i < parts; i += 32) dm += partial[i];
    dm = dev::warp_sum(dm);
    return (1.0 - d) / double(V) + d * dm / double(V);
}

// The graph's pull tasks (graph.cuh): a chunk of a long row gives its partial
// sum, a tile its rows' contributions, 32 rows at a time.  Three quarters of
// the tasks are dealt to the warps in turn, the others taken from `cursor`.
// Bound by the gathers, one L2 sector per in-edge: on R-MAT scale 22 (64 M
// edges) one warp per row and one per chunk took 1100 us, the tasks take 333 us.
constexpr int kContribThreads = 1024;

__global__ void __launch_bounds__(kContribThreads, 1) pagerank_contrib_kernel(
    const uint64_t *__restrict__ in_off, const uint32_t *__restrict__ in_src, const uint32_t *__restrict__ hot_vertex,
    uint32_t num_hot, const uint4 *__restrict__ tasks, uint64_t num_tasks, const LongRow *__restrict__ long_rows,
    const double *__restrict__ x, const float *__restrict__ rank, uint64_t V, double damping,
    const double *__restrict__ partial, int parts, uint32_t *cursor, double *__restrict__ chunk_sum,
    double *__restrict__ out) {
    extern __shared__ __align__(16) uint32_t s_hot[];
    __shared__ double s_share;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < num_hot; i += blockDim.x) s_hot[i] = hot_vertex[i];
    if (threadIdx.x < 32) {
        const double sh = base_share(partial, parts, V, damping, threadIdx.x);
        if (threadIdx.x == 0) s_share = sh;
    }
    __syncthreads();
    const double share = s_share;
    const uint64_t nwarps = uint64_t(gridDim.x) * (kContribThreads / 32);
    const uint64_t dealt = max(num_tasks - num_tasks / 4, min(num_tasks, nwarps));
    uint64_t task = uint64_t(blockIdx.x) * (kContribThreads / 32) + warp;
    while (task < num_tasks) {
        uint64_t next = task + nwarps;
        uint32_t ticket = 0;
        const bool ask = next >= dealt;
        if (ask && lane == 0) ticket = atomicAdd(cursor, 1u);
        const uint4 d = tasks[task];
        if (!ask) prefetch_task(tasks[next], in_src, nullptr, lane);
        const uint64_t e0 = task_first_edge(d);
        const InEdges E{in_src + e0, s_hot, x};
        if (task_is_chunk(d)) {
            const double acc = span_sum(E, 0, task_edges(d), lane);
            if (lane == 0) chunk_sum[long_rows[d.z].first_chunk + d.w] = acc;
        } else {
            for (uint32_t rb = d.z; rb < d.w; rb += 32) {
                const uint32_t r = rb + lane;
                uint32_t lo = 0, hi = 0;
                double old = 0.0;
                if (r < d.w) {
                    lo = static_cast<uint32_t>(in_off[r] - e0);
                    hi = static_cast<uint32_t>(in_off[r + 1] - e0);
                    old = rank[r];
                }
                const bool wide = hi - lo >= 64;
                const uint32_t hs = wide ? lo : hi;  // group steps see a wide row as empty
                const uint32_t most = __reduce_max_sync(0xffffffffu, hs - lo);
                double acc = 0.0;
                if (most > 32)
                    acc = group_sum<8, 8>(E, lo, hs, lane);
                else if (most > 16)
                    acc = group_sum<4, 8>(E, lo, hs, lane);
                else if (most > 8)
                    acc = group_sum<2, 8>(E, lo, hs, lane);
                else if (most > 4)
                    acc = group_sum<1, 8>(E, lo, hs, lane);
                else if (most)
                    acc = group_sum<1, 4>(E, lo, hs, lane);
                for (uint32_t big = __ballot_sync(0xffffffffu, wide); big; big &= big - 1) {
                    const int o = __ffs(big) - 1;
                    const double t = span_sum(E, __shfl_sync(0xffffffffu, lo, o), __shfl_sync(0xffffffffu, hi, o), lane);
                    if (lane == o) acc = t;
                }
                if (r < d.w) out[r] = fabs(share + damping * acc - old);
            }
        }
        if (ask) next = dealt + __shfl_sync(0xffffffffu, ticket, 0);
        task = next;
    }
}

// One warp per long row: its chunks' partial sums in a fixed order.
__global__ void contrib_long_rows_kernel(const LongRow *__restrict__ long_rows, uint64_t num_long,
                                         const double *__restrict__ chunk_sum, const float *__restrict__ rank,
                                         uint64_t V, double damping, const double *__restrict__ partial, int parts,
                                         double *__restrict__ out) {
    __shared__ double s_share;
    if (threadIdx.x < 32) {
        const double sh = base_share(partial, parts, V, damping, threadIdx.x);
        if (threadIdx.x == 0) s_share = sh;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const uint64_t warps = uint64_t(gridDim.x) * (blockDim.x >> 5);
    for (uint64_t i = (blockIdx.x * uint64_t(blockDim.x) + threadIdx.x) >> 5; i < num_long; i += warps) {
        const LongRow lr = long_rows[i];
        double acc = 0.0;
        for (uint32_t c = lane; c < lr.num_chunks; c += 32) acc += chunk_sum[lr.first_chunk + c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) out[lr.row] = fabs(s_share + damping * acc - double(rank[lr.row]));
    }
}

__global__ void sssp_contrib_kernel(const float *__restrict__ cur, const float *__restrict__ cand, uint64_t n,
                                    float tol, double *__restrict__ out) {
    for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < n; v += uint64_t(gridDim.x) * blockDim.x) {
        const float c = cur[v], d = cand[v];
        double r = 0.0;
        if (isfinite(c) && isfinite(d)) {
            const float improvement = __fsub_rn(c, d);
            if (improvement > tol) r = double(improvement);
        } else if (!isfinite(c) && isfinite(d)) {
            r = 1.0;
        }
        out[v] = r;
    }
}

// Order-preserving unsigned image of a finite double (-0 and +0 equal).
__device__ __forceinline__ uint64_t double_key(double c) {
    uint64_t b = static_cast<uint64_t>(__double_as_longlong(c == 0.0 ? 0.0 : c));
    return (b >> 63) ? ~b : (b | (uint64_t(1) << 63));
}

// What the host decides the sorts by.
struct ScheduleFacts {
    unsigned long long zero, nonfinite, moved, duplicates;  // metrics
    unsigned long long keys_or, keys_nand;                  // bits set in some key; bits clear in some key
    unsigned long long max_item;
    uint32_t descents;  // 1: some item does not exceed the one before it
    uint32_t pad;
};

// Keys and positions in input order, the zero and non-finite counts, which
// key bits differ, and whether the items ascend strictly.
__global__ void schedule_prep_kernel(const uint64_t *__restrict__ item, const double *__restrict__ c, uint64_t n,
                                     double eps, uint64_t *__restrict__ key, uint32_t *__restrict__ pos,
                                     ScheduleFacts *__restrict__ f) {
    unsigned long long zero = 0, nonfinite = 0, ones = 0, zeros = 0, top = 0;
    uint32_t descents = 0;
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x) {
        const double x = c[i];
        const uint64_t k = double_key(x), it = item[i];
        key[i] = k;
        pos[i] = static_cast<uint32_t>(i);
        if (!isfinite(x)) ++nonfinite;
        if (fabs(x) <= eps) ++zero;
        ones |= k;
        zeros |= ~k;
        top = max(top, static_cast<unsigned long long>(it));
        if (i && it <= item[i - 1]) descents = 1;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        zero += __shfl_xor_sync(0xffffffffu, zero, o);
        nonfinite += __shfl_xor_sync(0xffffffffu, nonfinite, o);
        ones |= __shfl_xor_sync(0xffffffffu, ones, o);
        zeros |= __shfl_xor_sync(0xffffffffu, zeros, o);
        top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    descents = __reduce_or_sync(0xffffffffu, descents);
    if ((threadIdx.x & 31) == 0) {
        if (zero) atomicAdd(&f->zero, zero);
        if (nonfinite) atomicAdd(&f->nonfinite, nonfinite);
        atomicOr(&f->keys_or, ones);
        atomicOr(&f->keys_nand, zeros);
        atomicMax(&f->max_item, top);
        if (descents) atomicOr(&f->descents, 1u);
    }
}

__global__ void contribution_keys_kernel(const double *__restrict__ c, const uint32_t *__restrict__ pos, uint64_t n,
                                         uint64_t *__restrict__ key) {
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        key[i] = double_key(c[pos[i]]);
}

__global__ void positions_kernel(uint32_t *pos, uint64_t n) {
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        pos[i] = static_cast<uint32_t>(i);
}

// ordered[p] = item[order[p]]; counts moved positions.
__global__ void schedule_emit_kernel(const uint64_t *__restrict__ item, const uint32_t *__restrict__ order, uint64_t n,
                                     uint64_t *__restrict__ ordered, ScheduleFacts *__restrict__ f) {
    unsigned long long moved = 0;
    for (uint64_t p = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; p < n; p += uint64_t(gridDim.x) * blockDim.x) {
        const uint64_t o = order[p];
        ordered[p] = item[o];
        moved += o != p;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) moved += __shfl_xor_sync(0xffffffffu, moved, o);
    if ((threadIdx.x & 31) == 0 && moved) atomicAdd(&f->moved, moved);
}

// Counts adjacent equal item indices in the sorted copy.
__global__ void duplicates_kernel(const uint64_t *__restrict__ sorted, uint64_t n, ScheduleFacts *f) {
    unsigned long long dup = 0;
    for (uint64_t i = 1 + blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        dup += sorted[i] == sorted[i - 1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dup += __shfl_xor_sync(0xffffffffu, dup, o);
    if ((threadIdx.x & 31) == 0 && dup) atomicAdd(&f->duplicates, dup);
}

unsigned grid_sm(unsigned per_sm) { return static_cast<unsigned>(sm_count()) * per_sm; }

// Stable radix sort of (key, value) pairs on key bits [first, bits).
template <class K, class V>
void sort_pairs(K *&keys, K *keys_alt, V *&vals, V *vals_alt, uint64_t n, bool descending, cudaStream_t s,
                int first, int bits) {
    if (n < 2 || first >= bits) return;
    cub::DoubleBuffer<K> kb(keys, keys_alt);
    cub::DoubleBuffer<V> vb(vals, vals_alt);
    size_t tb = 0;
    if (descending) {
        HYT_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tb, kb, vb, static_cast<int64_t>(n), first, bits, s));
    } else {
        HYT_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, kb, vb, static_cast<int64_t>(n), first, bits, s));
    }
    Scratch<uint8_t> tmp(tb, s);
    if (descending) {
        HYT_CUDA(cub::DeviceRadixSort::SortPairsDescending(tmp.get(), tb, kb, vb, static_cast<int64_t>(n), first, bits, s));
    } else {
        HYT_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), tb, kb, vb, static_cast<int64_t>(n), first, bits, s));
    }
    keys = kb.Current();
    vals = vb.Current();
}

}  // namespace

void pagerank_contributions(GraphImpl &g, const float *ranks, float damping, double *out, double *device_ms) {
    graph_require_caller_order(g, "hyt_pagerank_contributions");
    if (!(g.flags & HYT_GRAPH_PULL)) fail(HYT_E_INVALID, "graph was created without HYT_GRAPH_PULL");
    if (!ranks || !out) fail(HYT_E_INVALID, "NULL argument");
    if (!(damping >= 0.0f && damping < 1.0f)) fail(HYT_E_INVALID, "PageRank damping_factor must be in [0, 1)");
    const uint64_t V = g.V;
    if (V == 0) fail(HYT_E_INVALID, "PageRank requires at least one vertex");
    HYT_CUDA(cudaSetDevice(g.device));
    cudaStream_t s = g.stream;
    std::unique_ptr<Scratch<float>> rh;
    const float *r = device_view(ranks, V, rh, s);
    const bool out_dev = is_device_pointer(out);
    std::unique_ptr<Scratch<double>> oh;
    double *o = out;
    if (!out_dev) {
        oh = std::make_unique<Scratch<double>>(V, s);
        o = oh->get();
    }
    Scratch<double> partial(kPartBlocks + 1, s), x(V, s);
    uint32_t *cursor = reinterpret_cast<uint32_t *>(partial.get() + kPartBlocks);
    const uint64_t chunks = g.num_long ? g.num_chunks : 0;
    Scratch<double> chunk_sum(chunks ? chunks : 1, s);
    const unsigned smem = static_cast<unsigned>(g.num_hot * sizeof(uint32_t));
    if (smem > 32 * 1024)  // beyond what every kernel may have
        HYT_CUDA(cudaFuncSetAttribute(pagerank_contrib_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kPRSmemMax)));
    // blocks beyond the vertices would add zeros
    const int parts = static_cast<int>(std::min<uint64_t>(kPartBlocks, (V + 255) / 256));
    EventTimer t;
    t.start(s);
    source_shares_kernel<<<parts, 256, 0, s>>>(g.out_degree.get(), r, V, x.get(), partial.get(), cursor);
    // no more CTAs than have tasks: each loads the hot table
    const uint64_t want = (g.num_chunks + g.num_tiles + kContribThreads / 32 - 1) / (kContribThreads / 32);
    pagerank_contrib_kernel<<<static_cast<unsigned>(std::min<uint64_t>(grid_sm(1), want)), kContribThreads, smem, s>>>(
        g.in_offsets.get(), g.in_sources.get(), g.hot_vertex.get(), g.num_hot, g.pull_tasks.get(),
        g.num_chunks + g.num_tiles, g.long_rows.get(), x.get(), r, V, double(damping), partial.get(), parts,
        cursor, chunk_sum.get(), o);
    if (chunks) {
        contrib_long_rows_kernel<<<grid_for(g.num_long * 32, 256), 256, 0, s>>>(
            g.long_rows.get(), g.num_long, chunk_sum.get(), r, V, double(damping), partial.get(), parts, o);
    }
    HYT_CUDA(cudaGetLastError());
    t.stop(s);
    if (!out_dev) HYT_CUDA(cudaMemcpyAsync(out, o, V * 8, cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaStreamSynchronize(s));
    if (device_ms) *device_ms = t.ms();
}

void sssp_contributions(const float *cur, const float *cand, uint64_t n, float tol, double *out) {
    if (n && (!cur || !cand || !out)) fail(HYT_E_INVALID, "NULL argument");
    if (!(tol >= 0.0f) || !std::isfinite(tol))
        fail(HYT_E_INVALID, "SSSP contribution tolerance must be finite and non-negative");
    if (n == 0) return;
    StreamHold st;
    cudaStream_t s = st.s;
    std::unique_ptr<Scratch<float>> ch, dh;
    const float *c = device_view(cur, n, ch, s);
    const float *d = device_view(cand, n, dh, s);
    const bool out_dev = is_device_pointer(out);
    std::unique_ptr<Scratch<double>> oh;
    double *o = out;
    if (!out_dev) {
        oh = std::make_unique<Scratch<double>>(n, s);
        o = oh->get();
    }
    sssp_contrib_kernel<<<grid_for(n, 256), 256, 0, s>>>(c, d, n, tol, o);
    HYT_CUDA(cudaGetLastError());
    if (!out_dev) HYT_CUDA(cudaMemcpyAsync(out, o, n * 8, cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaStreamSynchronize(s));
}

void contribution_schedule(const uint64_t *item, const double *contribution, uint64_t n, bool deterministic,
                           double eps, uint64_t *ordered, hyt_contribution_metrics *m) {
    if (!m) fail(HYT_E_INVALID, "metrics is NULL");
    std::memset(m, 0, sizeof(*m));
    if (n && (!item || !contribution || !ordered)) fail(HYT_E_INVALID, "NULL argument");
    m->input_item_count = n;
    m->scheduled_item_count = n;
    if (n == 0) return;
    StreamHold st;
    cudaStream_t s = st.s;
    std::unique_ptr<Scratch<uint64_t>> ih;
    std::unique_ptr<Scratch<double>> chold;
    const uint64_t *it = device_view(item, n, ih, s);
    const double *c = device_view(contribution, n, chold, s);
    if (n > 0xFFFFFFFFull) fail(HYT_E_OOM, "contribution schedules hold fewer than 2^32 items");
    const bool ordered_dev = is_device_pointer(ordered);
    Scratch<uint32_t> pos(n, s), pos_alt(n, s);
    Scratch<uint64_t> key(n, s), key_alt(n, s), out_d(ordered_dev ? 1 : n, s);
    Scratch<ScheduleFacts> facts(1, s);
    HYT_CUDA(cudaMemsetAsync(facts.get(), 0, sizeof(ScheduleFacts), s));
    schedule_prep_kernel<<<grid_for(n, 256, 148u * 8u), 256, 0, s>>>(it, c, n, eps, key.get(), pos.get(), facts.get());
    HYT_CUDA(cudaGetLastError());
    ScheduleFacts h{};
    HYT_CUDA(cudaMemcpyAsync(&h, facts.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaStreamSynchronize(s));
    if (h.nonfinite) fail(HYT_E_INVALID, "contribution priority must be finite");
    uint32_t *vp = pos.get(), *vp_alt = pos_alt.get();
    uint64_t *ck = key.get(), *ck_alt = key_alt.get();
    // Items that ascend strictly (the vertices of a graph, say) are in item
    // order already and hold no duplicates; others are sorted for both, on
    // the bits the largest item needs.
    if (h.descents) {
        const int item_bits = h.max_item ? 64 - __builtin_clzll(h.max_item) : 1;
        Scratch<uint64_t> ik(n, s), ik_alt(n, s);
        uint64_t *ip = ik.get();
        HYT_CUDA(cudaMemcpyAsync(ip, it, n * 8, cudaMemcpyDeviceToDevice, s));
        sort_pairs(ip, ik_alt.get(), vp, vp_alt, n, false, s, 0, item_bits);
        duplicates_kernel<<<grid_for(n, 256, 148u * 8u), 256, 0, s>>>(ip, n, facts.get());
        HYT_CUDA(cudaGetLastError());
        if (deterministic) {
            vp_alt = vp == pos.get() ? pos_alt.get() : pos.get();
            contribution_keys_kernel<<<grid_for(n, 256, 148u * 8u), 256, 0, s>>>(c, vp, n, ck);
            HYT_CUDA(cudaGetLastError());
        } else {  // ties stay in input order
            vp = pos.get();
            vp_alt = pos_alt.get();
            positions_kernel<<<grid_for(n, 256, 148u * 8u), 256, 0, s>>>(vp, n);
            HYT_CUDA(cudaGetLastError());
        }
    }
    // by descending contribution, over the key bits that differ at all
    // (contributions that are differences of floats leave the low 29 alone)
    const unsigned long long differ = h.keys_or & h.keys_nand;
    if (differ)
        sort_pairs(ck, ck_alt, vp, vp_alt, n, true, s, __builtin_ctzll(differ), 64 - __builtin_clzll(differ));
    uint64_t *od = ordered_dev ? ordered : out_d.get();
    schedule_emit_kernel<<<grid_for(n, 256, 148u * 8u), 256, 0, s>>>(it, vp, n, od, facts.get());
    HYT_CUDA(cudaGetLastError());
    if (!ordered_dev) HYT_CUDA(cudaMemcpyAsync(ordered, od, n * 8, cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaMemcpyAsync(&h, facts.get(), sizeof(h), cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaStreamSynchronize(s));
    m->zero_contribution_count = h.zero;
    m->reordered_item_count = h.moved;
    m->redundant_work_count = h.duplicates;
    m->scheduling_overhead = std::log2(static_cast<double>(n));
}

void partition_contributions(const double *contrib, uint64_t V, const uint64_t *bounds, uint64_t parts, double *out) {
    if (parts && (!bounds || !out)) fail(HYT_E_INVALID, "NULL argument");
    if (V && !contrib) fail(HYT_E_INVALID, "NULL argument");
    if (parts == 0) return;
    StreamHold st;
    cudaStream_t s = st.s;
    std::unique_ptr<Scratch<double>> ch;
    std::unique_ptr<Scratch<uint64_t>> bh;
    std::vector<uint64_t> hb(parts + 1);
    HYT_CUDA(cudaMemcpyAsync(hb.data(), bounds, (parts + 1) * 8, cudaMemcpyDefault, s));
    HYT_CUDA(cudaStreamSynchronize(s));
    for (uint64_t i = 0; i < parts; ++i)
        if (hb[i] > hb[i + 1] || hb[i + 1] > V) fail(HYT_E_INVALID, "partition bounds must be non-decreasing and <= V");
    const double *c = device_view(contrib, V, ch, s);
    const uint64_t *b = device_view(bounds, parts + 1, bh, s);
    const bool out_dev = is_device_pointer(out);
    std::unique_ptr<Scratch<double>> oh;
    double *o = out;
    if (!out_dev) {
        oh = std::make_unique<Scratch<double>>(parts, s);
        o = oh->get();
    }
    size_t tb = 0;
    HYT_CUDA(cub::DeviceSegmentedReduce::Sum(nullptr, tb, c, o, static_cast<int64_t>(parts), b, b + 1, s));
    Scratch<uint8_t> tmp(tb, s);
    HYT_CUDA(cub::DeviceSegmentedReduce::Sum(tmp.get(), tb, c, o, static_cast<int64_t>(parts), b, b + 1, s));
    if (!out_dev) HYT_CUDA(cudaMemcpyAsync(out, o, parts * 8, cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaStreamSynchronize(s));
}

}  // namespace hyt
