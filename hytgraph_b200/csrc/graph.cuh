// Device-resident graph behind the opaque hyt_graph handle.
//
// HBM layout (E < 2^32 edges per graph on this path):
//   push side (CSR, frontier SSSP):   row_offsets u64[V+1], cols u32[E],
//                                     weights u32[E] (u32 or f32 bits)
//   pull side (CSC, PageRank):        in_offsets u64[V+1], in_sources u32[E]
//   per vertex:                       out_degree u32[V]
//   PageRank work list:               tile_start u32[T+1] (short-row tiles),
//                                     long rows + their chunk tasks
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <vector>

#include "common.cuh"

namespace hyt {

// PageRank pull work decomposition.  Rows are cut into tiles along the
// merge path (1 unit per row + 1 per in-edge): a tile spans tile_cost units,
// so its rows hold fewer than tile_cost edges except for its last row.  A
// last row with in-degree >= tile_cost is a "long row": it is excluded from
// the tile and split into chunks.  One warp processes one task (tile or
// chunk).
constexpr uint32_t kTileCostMin = 64;
constexpr uint32_t kTileCostSmall = 512;     // ... on small ones
constexpr uint32_t kTileCostDefault = 1024;  // merge-path units per tile on large graphs (tunable: HYT_PR_TILE)
constexpr uint32_t kStageTileMax = 256;      // bulk-staged kernels: a tile's edges (< 2 * tile_cost) fit one slot
// Edges per chunk of a long row.  A warp takes a chunk 256 edges at a time, so a
// chunk is also the longest serial chain of a pass: 4096 edges cost 25 us, which
// small graphs and out-of-HBM pieces have no other work to hide, while on large
// graphs every chunk more is a hand-over more.  Measured with 1024 / 2048 / 4096
// edges: PageRank on 131 K vertices, 2 M edges 468 / 500 / 598 us; on 1 M, 17 M
// 1254 / 1121 / 1122 us; eight packed PPRs on 2 M, 34 M 5.13 / 5.17 / 5.39 ms;
// PageRank on 16 M, 263 M 17.9 / 17.2 / 16.9 ms.
constexpr uint32_t kLongChunkSmall = 1024;
constexpr uint32_t kLongChunk = 4096;
inline uint32_t long_chunk_edges(uint64_t rows_and_edges) {
    if (rows_and_edges < uint64_t(1) << 23) return kLongChunkSmall;
    return rows_and_edges < uint64_t(1) << 26 ? 2048u : kLongChunk;
}
constexpr uint32_t kHotSourcesDefault = 8192;   // shared-memory source cache (tunable: HYT_PR_HOT)
constexpr uint32_t kHotSourcesLarge = 24576;    // ... of graphs of kHotLargeVertices or more
constexpr uint64_t kHotLargeVertices = uint64_t(1) << 22;  // PageRank 8192 -> 24576 entries: 18.45 -> 17.75 ms at 2^24 vertices,
                                                           // 4.58 -> 4.52 at 2^22; 1.43 -> 1.53 at 2^20 (loading them costs more)
constexpr uint32_t kHotSourcesMax = 32768;
constexpr uint32_t kPRSmemMax = 226 * 1024;     // dynamic shared memory per CTA (227 KB opt-in - static)
constexpr uint32_t kHotTag = 0x80000000u;       // in_sources tag: source is hot slot (low bits)

// Pull task descriptors (pull_tasks[i], chunks first, then tiles: the task
// numbering of the pull kernels), 16 bytes each so a warp fetches its next
// task with one load:
//   x = first edge (low 32 bits)
//   y = first edge bits 32..39 | edge count << 8 (< 2^23) | 1 << 31 for a chunk
//   z, w = first row and end row of a tile (the end excludes a chunked long
//          last row); long-row index and chunk number of a chunk
__host__ __device__ __forceinline__ uint64_t task_first_edge(uint4 d) {
    return uint64_t(d.x) | (uint64_t(d.y & 0xFFu) << 32);
}
__host__ __device__ __forceinline__ uint32_t task_edges(uint4 d) { return (d.y >> 8) & 0x7FFFFFu; }
__host__ __device__ __forceinline__ bool task_is_chunk(uint4 d) { return (d.y >> 31) != 0; }

#ifndef HYT_PULL_PREFETCH
#define HYT_PULL_PREFETCH 1
#endif
#ifdef __CUDACC__
// Warms L2 with the edge arrays a0 (and a1 when not NULL) of pull task d:
// lane l touches the 128-byte lines at edges l*32, l*32 + 1024, ... of the
// task, so the next task's streaming loads find their lines in L2.
__device__ __forceinline__ void prefetch_task(uint4 d, const uint32_t *a0, const uint32_t *a1, int lane) {
    if constexpr (HYT_PULL_PREFETCH) {
        const uint64_t e0 = task_first_edge(d), n = task_edges(d);
        for (uint64_t x = uint64_t(lane) * 32; x < n; x += 32 * 32) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a0 + e0 + x));
            if (a1) asm volatile("prefetch.global.L2 [%0];" ::"l"(a1 + e0 + x));
        }
    }
}
#endif

struct LongRow {
    uint32_t row;
    uint32_t first_chunk;  // index of its first partial-sum slot
    uint32_t num_chunks;
    uint32_t pad;
};

// An instantiated CUDA graph holding a solver's conditional while-loop,
// kept with the graph object and reused by later solves while the loop's
// shape (`key`: kernels, launch shapes, argument pointers) is unchanged.
// Its conditional handle is set to 1 at every launch.
struct LoopGraph {
    std::vector<unsigned char> key;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaGraphConditionalHandle cond = 0;

    LoopGraph() = default;
    LoopGraph(const LoopGraph &) = delete;
    LoopGraph &operator=(const LoopGraph &) = delete;
    ~LoopGraph() { reset(); }
    void reset() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
        key.clear();
    }
    bool matches(const void *k, size_t n) const {
        return exec && key.size() == n && std::memcmp(key.data(), k, n) == 0;
    }
    void set_key(const void *k, size_t n) {
        key.assign(static_cast<const unsigned char *>(k), static_cast<const unsigned char *>(k) + n);
    }
};

// Two side streams of a call and the events that fork and join them, kept with
// the graph: made and destroyed by each call they cost 0.2 ms.
struct SideStreams {
    cudaStream_t stream[2] = {};
    cudaEvent_t fork = nullptr, join[2] = {};
    SideStreams() = default;
    SideStreams(const SideStreams &) = delete;
    SideStreams &operator=(const SideStreams &) = delete;
    void open() {
        if (!fork) HYT_CUDA(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
        for (int i = 0; i < 2; ++i) {
            if (!stream[i]) HYT_CUDA(cudaStreamCreateWithFlags(&stream[i], cudaStreamNonBlocking));
            if (!join[i]) HYT_CUDA(cudaEventCreateWithFlags(&join[i], cudaEventDisableTiming));
        }
    }
    // waits for their work
    void settle() noexcept {
        for (cudaStream_t s : stream)
            if (s) cudaStreamSynchronize(s);
    }
    ~SideStreams() {
        settle();
        for (int i = 0; i < 2; ++i) {
            if (stream[i]) cudaStreamDestroy(stream[i]);
            if (join[i]) cudaEventDestroy(join[i]);
        }
        if (fork) cudaEventDestroy(fork);
    }
};

// Smallest and largest weight (bit patterns, sign of -0.0 cleared).
struct WeightRange {
    uint32_t low = 0, high = 0;
};

struct GraphImpl {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;

    uint64_t V = 0, E = 0;
    uint32_t weight_kind = HYT_WEIGHTS_NONE;
    uint32_t flags = 0;
    bool weights_ok = true;  // F32 weights all finite and >= 0
    uint32_t default_delta = 0;  // SSSP near/far bucket width (2x mean u32 weight)

    // push side
    GraphArray<uint64_t> row_offsets;
    GraphArray<uint32_t> cols;
    GraphArray<uint32_t> weights;
    GraphArray<uint32_t> out_degree;
    // HYT_GRAPH_HUB_ORDER: perm[new] = caller id, inv[caller id] = new
    // (empty otherwise)
    GraphArray<uint32_t> perm, inv;
    std::vector<uint32_t> h_inv;  // host copy of inv, filled by graph_vertex_map (engines mapping many sources)

    // pull side
    GraphArray<uint64_t> in_offsets;
    GraphArray<uint32_t> in_sources;
    // [E] weights in CSC order (PUSH|PULL weighted graphs; SSSP pull rounds).
    // in_pack_bits > 0: (source id | weight << in_pack_bits) in one word, with
    // which a sweep loads one stream in place of two and looks up no hot slot.
    GraphArray<uint32_t> in_weights;
    uint32_t in_pack_bits = 0;
    GraphArray<uint32_t> tile_start;   // [num_tiles + 1]
    GraphArray<LongRow> long_rows;     // [num_long]
    GraphArray<uint2> chunk_tasks;     // [num_chunks] = (long row index, chunk)
    GraphArray<uint4> pull_tasks;      // [num_chunks + num_tiles] descriptors (task_first_edge, ...)
    uint64_t num_tiles = 0, num_long = 0, num_chunks = 0;
    uint32_t tile_cost = kTileCostDefault;  // a row is long when its in-degree >= tile_cost
    uint32_t chunk_edges = kLongChunk;      // edges per chunk of a long row
    // Hot sources: the num_hot vertices of largest out-degree.  Their
    // occurrences in in_sources carry kHotTag | slot, and each PageRank CTA
    // keeps their contributions in shared memory for the iteration.
    GraphArray<uint32_t> hot_vertex;   // [num_hot], by slot
    uint32_t num_hot = 0;
    uint64_t hot_edges = 0;             // in-edges whose source is hot

    // host-side facts
    uint64_t max_in_degree = 0, max_out_degree = 0, dangling = 0;
    double build_ms = 0.0;

    // Solver workspaces, grown on demand and reused across calls.
    GraphArray<float> rank[2];
    GraphArray<float> contrib[2];
    GraphArray<float> partial;        // long-row chunk partial sums (s, c)
    GraphArray<uint32_t> ticket;      // long-row arrival counters
    GraphArray<unsigned char> pr_state;

    GraphArray<uint32_t> dist;
    GraphArray<uint32_t> stamp;
    GraphArray<uint32_t> queue[2];
    GraphArray<uint32_t> far[2];
    GraphArray<uint2> hub_tasks;
    GraphArray<unsigned char> sssp_state;
    GraphArray<uint32_t> ppr_wide;         // packed PPR: rows of 32+ in-edges below the long-row threshold
    uint64_t ppr_wide_n = 0;
    bool ppr_wide_ready = false;
    WeightRange weight_range;              // of the weights kept
    GraphArray<uint32_t> ms_dist;          // multi-source labels [V][8]
    GraphArray<unsigned char> ms_state;
    PinnedArray<uint64_t> host_scratch;  // small pinned readback area
    LoopGraph sssp_loop;                 // instantiated SSSP round loop (reused while its shape holds)
    LoopGraph ms_loop;                   // ... of the multi-source solve
    SideStreams side;                    // packed PPR: two of the three row classes

    size_t device_bytes() const;
};

// PageRank CTA shape: kPRThreads threads; dynamic shared memory = hot
// cache and its zero slot.
constexpr int kPRThreads = 1024;
inline size_t pr_hot_bytes(uint32_t num_hot) { return (size_t(num_hot) + 1) * sizeof(float); }
// Pull tasks that a whole-graph pass deals to the warps in turn; the others are
// taken one by one by whichever warp is free, at the price of an atomic and a
// descriptor read that nothing hides.  Tasks of a graph in input order cost
// uneven amounts (rows of all degrees side by side): a quarter handed out takes
// PageRank on 16.7 M vertices from 22.9 to 20.1 ms and on 0.5 M from 0.95 to
// 0.85 ms.  In hub order neighbours are alike: 17.3 -> 16.9 ms at 16.7 M, but
// 1.09 -> 1.22 ms at 1 M, where a warp has 4 tasks in all.
inline uint64_t dealt_tasks(const GraphImpl &g) {
    const uint64_t n = g.num_chunks + g.num_tiles;
    const bool even = g.perm.get() && n < 16ull * sm_count() * (kPRThreads / 32);
    return even ? n : n - n / 4;
}

// Merge-path units per tile of a graph (graph.cu).
uint32_t tile_cost_for(uint64_t V, uint64_t E);

// Builds the device graph from a CSR (host or device pointers).
void graph_build(GraphImpl &g, const hyt_csr &csr, uint32_t flags);

// Copies the CSC with hot tags removed into caller buffers (host or device).
void graph_copy_csc(const GraphImpl &g, uint64_t *in_offsets, uint32_t *in_sources);
// Builds the graph; with HYT_GRAPH_HUB_ORDER in flags, in hub order.
void graph_create(GraphImpl &g, const hyt_csr &csr, uint32_t flags);
// The internal id of a caller's vertex (identity without a hub order):
// from the host copy of the map when graph_vertex_map has made one, else
// one 4-byte read of the device map on stream s.
uint32_t graph_vertex(const GraphImpl &g, uint32_t v, cudaStream_t s);
// Makes the host copy of a hub-ordered graph's vertex map (once), for
// callers that map many sources; no-op without a hub order.
void graph_vertex_map(GraphImpl &g);
// Writes V 4-byte per-vertex values (internal order, device) to dst (host
// or device) in the caller's vertex order.
void graph_emit(const GraphImpl &g, void *dst, const void *src, cudaStream_t s);
// Fails with HYT_E_UNSUPPORTED for a hub-ordered graph.
void graph_require_caller_order(const GraphImpl &g, const char *what);

}  // namespace hyt

struct hyt_graph {
    hyt::GraphImpl impl;
};
