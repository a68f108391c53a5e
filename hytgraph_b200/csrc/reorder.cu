// Hub-vertex sorting and vertex reordering on the GPU (hyt_hub_sort,
// hyt_csr_reorder).
//
// Hub sort follows the reference's HubSorter::sort
// (src/scheduling/hub_sort.cpp:28-183):
//   H(v) = Do(v) * Di(v) / (Do_max * Di_max),
//   hub_count = round(V * fraction) when V * fraction is within 1e-12 of an
//               integer, else ceil(V * fraction), capped at V,
//   the hub_count highest scores first (ties: lower vertex id first), then
//   every other vertex in its original relative order.
// Scores equal the reference's bit for bit: its long-double quotient is
// the x86-64 extended format (64-bit significand), which the kernel
// reproduces with an exact integer long division rounded to 64 bits and then
// to 53 bits, both to nearest-even.  The ranking sorts those doubles' bit
// patterns (non-negative doubles order like their bits), or the degree
// products where these rank alike, with a stable descending radix sort over
// ids in ascending order, which is the reference's comparator.
//
// Reordering follows CSRGraph::reorder_vertices
// (src/graph/csr_graph.cpp:171-283): vertex_order[new] = old; new row
// `new` holds old row `old`'s edges in their original order, destinations
// renamed through the inverse permutation, weights carried along.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <unordered_map>

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include "common.cuh"
#include "outputs.cuh"
#include "scratch.cuh"
#include "solvers.cuh"

namespace hyt {
namespace {

using dev::ld_stream;
using dev::policy_evict_last;

// Read-only 32-bit gather with an L2 eviction policy (no volatile: the
// compiler may batch independent gathers).
__device__ __forceinline__ uint32_t ld_nc_keep(const uint32_t *p, uint64_t pol) {
    uint32_t v;
    asm("ld.global.nc.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
    return v;
}

enum : uint32_t {
    kBadOffsets = 1u,     // offsets do not start at 0 or decrease
    kBadTerminal = 2u,    // last offset != E
    kBadColumn = 4u,      // destination >= V
    kBadOrderRange = 8u,  // vertex_order entry >= V
    kBadOrderDup = 16u,   // vertex_order entry repeated
    kBadOverflow = 32u,   // Do_max * Di_max >= 2^64
};

__device__ __forceinline__ uint64_t warp_max_u64(uint64_t x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = max(x, __shfl_xor_sync(0xffffffffu, x, o));
    return x;
}

// One pass over the CSR: in-degrees, out-degrees, the largest out-degree, and
// the structure checks of the reference's CSRGraph::validate (offsets start
// at 0, never decrease, end at E; every destination is a vertex).
//
// Plain global atomics were bound by the hub destinations, whose additions
// queue up at one address each (671 us on R-MAT scale 22, 58 M edges).  Every
// CTA therefore counts in a small direct-mapped table in shared memory first:
// the first destination to come by a slot keeps it -- most likely the most
// frequent of those that share it -- and the others go to global memory: 536
// us.
constexpr int kDegreeThreads = 1024;
constexpr uint32_t kDegreeSlots = 8192;
constexpr int kDegreeUnroll = 4;

__global__ void __launch_bounds__(kDegreeThreads, 2) degree_pass_kernel(
    const uint64_t *__restrict__ off, const uint32_t *__restrict__ cols, uint64_t V, uint64_t E,
    uint32_t *__restrict__ indeg, uint64_t *__restrict__ outdeg, unsigned long long *__restrict__ maxes,
    uint32_t *__restrict__ bad) {
    extern __shared__ uint32_t s_tab[];
    uint32_t *s_key = s_tab, *s_cnt = s_tab + kDegreeSlots;
    constexpr uint32_t kFree = 0xFFFFFFFFu;  // no destination: ids are below V < 2^32
    for (uint32_t i = threadIdx.x; i < kDegreeSlots; i += kDegreeThreads) {
        s_key[i] = kFree;
        s_cnt[i] = 0;
    }
    __syncthreads();
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    const uint64_t tid = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    uint32_t b = 0;
    for (uint64_t e = tid; e < E; e += kDegreeUnroll * stride) {
        uint32_t c[kDegreeUnroll];
#pragma unroll
        for (int j = 0; j < kDegreeUnroll; ++j) c[j] = e + j * stride < E ? ld_stream(cols + e + j * stride) : kFree;
#pragma unroll
        for (int j = 0; j < kDegreeUnroll; ++j) {
            if (e + j * stride >= E) continue;
            if (c[j] >= V) {
                b |= kBadColumn;
                continue;
            }
            const uint32_t slot = (c[j] * 2654435761u) >> 19;  // top 13 bits
            uint32_t k = *reinterpret_cast<volatile uint32_t *>(s_key + slot);
            if (k == kFree) {
                k = atomicCAS(s_key + slot, kFree, c[j]);
                if (k == kFree) k = c[j];
            }
            if (k == c[j])
                atomicAdd(s_cnt + slot, 1u);
            else
                atomicAdd(indeg + c[j], 1u);
        }
    }
    uint64_t mo = 0;
    for (uint64_t v = tid; v < V; v += stride) {
        const uint64_t a = off[v], z = off[v + 1];
        uint64_t d = 0;
        if (z < a) {
            b |= kBadOffsets;
        } else {
            d = z - a;
        }
        outdeg[v] = d;
        mo = max(mo, d);
    }
    if (tid == 0) {
        if (off[0] != 0) b |= kBadOffsets;
        if (off[V] != E) b |= kBadTerminal;
    }
    mo = warp_max_u64(mo);
    if ((threadIdx.x & 31) == 0 && mo) atomicMax(maxes, static_cast<unsigned long long>(mo));
    if (b) atomicOr(bad, b);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kDegreeSlots; i += kDegreeThreads)
        if (s_cnt[i]) atomicAdd(indeg + s_key[i], s_cnt[i]);
}

__global__ void max_in_degree_kernel(const uint32_t *__restrict__ indeg, uint64_t V, unsigned long long *maxes) {
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    uint64_t m = 0;
    for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < V; v += stride) m = max(m, uint64_t(indeg[v]));
    m = warp_max_u64(m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(maxes + 1, static_cast<unsigned long long>(m));
}

// n / d for 0 < n <= d < 2^64, rounded first to a 64-bit significand and
// then to a double, both to nearest-even: what x86-64 gives for
// (double)((long double)n / (long double)d).
__device__ double extended_quotient(uint64_t n, uint64_t d) {
    const int cn = __clzll(static_cast<long long>(n)), cd = __clzll(static_cast<long long>(d));
    const uint64_t a = n << cn, b = d << cd;  // both in [2^63, 2^64)
    // q = floor(a * 2^s / b) in [2^63, 2^64), s = 63 when a >= b else 64
    int s = 64;
    uint64_t q = 0, r = a;
    if (a >= b) {
        q = 1;
        r = a - b;
        s = 63;
    }
    for (int i = 0; i < s; ++i) {
        const bool carry = (r >> 63) != 0;
        r <<= 1;
        q <<= 1;
        if (carry || r >= b) {
            r -= b;
            q |= 1;
        }
    }
    int e = cd - cn - s;  // n / d = (q + r / b) * 2^e
    const uint64_t rest = b - r;
    if (r > rest || (r == rest && (q & 1))) {
        if (++q == 0) {
            q = uint64_t(1) << 63;
            ++e;
        }
    }
    const uint64_t low = q & 0x7FF;  // drop 11 bits: 64 -> 53
    uint64_t m = q >> 11;
    e += 11;
    if (low > 0x400 || (low == 0x400 && (m & 1))) {
        if (++m == (uint64_t(1) << 53)) {
            m >>= 1;
            ++e;
        }
    }
    // m * 2^e with m in [2^52, 2^53); e + 52 lies in [-64, 0]
    const uint64_t bits = (uint64_t(e + 52 + 1023) << 52) | (m & ((uint64_t(1) << 52) - 1));
    return __longlong_as_double(static_cast<long long>(bits));
}

// extended_quotient for 0 < n <= d < 2^52, from one IEEE division.  Rounding
// to 64 and then to 53 bits differs from rounding to 53 at once only where the
// 64-bit value is a 53-bit tie, so where the exact remainder shows the
// quotient within 2^-9 of half a unit from the double (or the double is a
// power of two, whose neighbours are unevenly spaced), the long division
// decides.
__device__ __forceinline__ double short_quotient(uint64_t n, uint64_t d) {
    const double x = static_cast<double>(n), y = static_cast<double>(d);
    const double q = __ddiv_rn(x, y);
    const double r = fabs(__fma_rn(-q, y, x));  // exact
    const uint64_t bits = static_cast<uint64_t>(__double_as_longlong(q));
    const double half = __longlong_as_double(static_cast<long long>(((bits >> 52) - 53) << 52)) * y;
    const bool sure = fabs(r - half) > half * 0x1p-9 && (bits << 12) != 0;
    return sure || r == 0.0 ? q : extended_quotient(n, d);
}

// Scores, ranking keys, and (each if asked for) which vertices have a score above
// 0 and the vertices' ids.  The
// denominator Do_max * Di_max is read from device memory (maxes[0..1]).
// Products below 2^52 rank exactly as their quotients do (two that differ are
// more than one unit in the last place apart after the division, so rounding
// keeps them apart), and have fewer bits to sort; above, the key is the
// score's bit pattern.
__device__ __forceinline__ bool rank_by_product(uint64_t denom) { return denom < (uint64_t(1) << 52); }

__global__ void hub_scores_kernel(const uint64_t *__restrict__ outdeg, const uint32_t *__restrict__ indeg, uint64_t V,
                                  const unsigned long long *__restrict__ maxes, double *__restrict__ scores,
                                  uint64_t *__restrict__ key, uint8_t *__restrict__ scored, uint32_t *__restrict__ id,
                                  uint32_t *__restrict__ bad) {
    const uint64_t max_out = maxes[0], max_in = maxes[1];
    const bool overflow = max_in && max_out > ~uint64_t(0) / max_in;
    if (overflow && blockIdx.x == 0 && threadIdx.x == 0) atomicOr(bad, kBadOverflow);
    const uint64_t denom = max_out * max_in;
    const bool product = !overflow && rank_by_product(denom);
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t v = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; v < V; v += stride) {
        const uint64_t num = outdeg[v] * uint64_t(indeg[v]);
        double sc = 0.0;
        if (num && !overflow && (scores || !product)) sc = product ? short_quotient(num, denom) : extended_quotient(num, denom);
        if (scores) scores[v] = sc;
        key[v] = product ? num : static_cast<uint64_t>(__double_as_longlong(sc));
        if (scored) scored[v] = num && !overflow;
        if (id) id[v] = static_cast<uint32_t>(v);
    }
}

// keys[i] = key[ids[i]]
__global__ void gather_keys_kernel(const uint64_t *__restrict__ key, const uint32_t *__restrict__ ids, uint64_t n,
                                   uint64_t *__restrict__ keys) {
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += stride) keys[i] = key[ids[i]];
}

__global__ void mark_kernel(const uint32_t *ids, uint64_t n, uint8_t *flag) {
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += stride) flag[ids[i]] = 0;
}

// Permutation check, inverse permutation (inv pre-filled with ~0: a second
// writer of the same old id is a duplicate), permuted degrees, and the
// offset checks.  ndeg[V] = 0 so an exclusive scan over V + 1 entries
// yields the new offsets.
__global__ void order_pass_kernel(const uint64_t *__restrict__ off, const uint32_t *__restrict__ order, uint64_t V,
                                  uint64_t E, uint32_t *__restrict__ inv, uint64_t *__restrict__ ndeg,
                                  uint32_t *__restrict__ bad) {
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    const uint64_t tid = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x;
    uint32_t b = 0;
    for (uint64_t nv = tid; nv < V; nv += stride) {
        const uint32_t old = order[nv];
        uint64_t d = 0;
        if (old >= V) {
            b |= kBadOrderRange;
        } else {
            if (atomicExch(inv + old, static_cast<uint32_t>(nv)) != 0xFFFFFFFFu) b |= kBadOrderDup;
            const uint64_t a = off[old], z = off[old + 1];
            if (z < a) {
                b |= kBadOffsets;
            } else {
                d = z - a;
            }
        }
        ndeg[nv] = d;
    }
    if (tid == 0) {
        if (off[0] != 0) b |= kBadOffsets;
        if (off[V] != E) b |= kBadTerminal;
        ndeg[V] = 0;
    }
    if (b) atomicOr(bad, b);
}

// Largest r < V with noff[r] <= e, for e < noff[V].
__device__ __forceinline__ uint64_t row_of(const uint64_t *__restrict__ noff, uint64_t V, uint64_t e) {
    uint64_t lo = 0, hi = V;  // noff[lo] <= e < noff[hi]
    while (hi - lo > 1) {
        const uint64_t mid = (lo + hi) >> 1;
        if (noff[mid] <= e) {
            lo = mid;
        } else {
            hi = mid;
        }
    }
    return lo;
}

constexpr int kPermThreads = 256;
constexpr int kPermEdges = 8;
constexpr uint64_t kTileEdges = uint64_t(kPermThreads) * kPermEdges;
constexpr uint32_t kTileRows = 2048;

// tile_row[t] = row holding the tile's first edge, for t < tiles;
// tile_row[tiles] = row holding the last edge.  Requires E > 0.
__global__ void tile_rows_kernel(const uint64_t *__restrict__ noff, uint64_t V, uint64_t E, uint64_t tiles,
                                 uint64_t *__restrict__ tile_row) {
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t t = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; t <= tiles; t += stride)
        tile_row[t] = row_of(noff, V, t < tiles ? t * kTileEdges : E - 1);
}

// New edge e of new row r copies old edge off[order[r]] + (e - noff[r]),
// destination renamed through inv, weight carried.  Tiles of 2048
// consecutive output edges; rows tile_row[t] .. tile_row[t + 1] cover the
// tile.  Each row's distance from new to old edge numbers is staged in shared
// memory, and each edge's row comes from a load-balanced search: every
// non-empty row marks its start inside the tile, and an inclusive max-scan
// over the 2048 positions hands each edge the last row starting at or before
// it.  A tile spanning more than 2048 rows (long runs of empty rows) searches
// the global offsets per edge instead.  Consecutive lanes take consecutive
// edges, so id / weight reads and writes are coalesced within a row; each
// thread keeps its 8 edges' loads in flight together (ids and weights, then
// the renaming gathers).
//
// The renaming gathers bound it, at the rate that the L1 beside shared memory
// allows (1.02 sectors per clock and SM with all of it, 0.28 beside 200 KB): 40
// KB of shared memory per CTA, five to an SM, held it to 771 us on R-MAT scale
// 22 (58 M edges); 20 KB take 484 us.
__global__ void __launch_bounds__(kPermThreads) permute_edges_kernel(
    const uint64_t *__restrict__ off, const uint32_t *__restrict__ cols, const uint32_t *__restrict__ w,
    const uint64_t *__restrict__ noff, const uint64_t *__restrict__ tile_row, const uint32_t *__restrict__ order,
    const uint32_t *__restrict__ inv, uint64_t V, uint64_t E, uint32_t *__restrict__ ncols,
    uint32_t *__restrict__ nw, uint32_t *__restrict__ bad) {
    __shared__ int64_t s_shift[kTileRows];  // old minus new edge number of row k's edges
    __shared__ __align__(16) uint16_t s_row[kTileEdges];
    __shared__ uint32_t s_warp[kPermThreads / 32];
    static_assert(kTileRows <= 65536 && kPermEdges == 8, "a thread scans 8 16-bit marks");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t b = 0;
    const uint64_t pol = policy_evict_last();
    const uint64_t tiles = (E + kTileEdges - 1) / kTileEdges;
    for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint64_t e0 = t * kTileEdges, e1 = min(e0 + kTileEdges, E);
        const uint64_t r0 = tile_row[t];
        const uint64_t rows = tile_row[t + 1] - r0 + 1;  // r0 + rows <= V
        const bool staged = rows <= kTileRows;
        if (staged) {
            reinterpret_cast<uint4 *>(s_row)[threadIdx.x] = make_uint4(0, 0, 0, 0);
            __syncthreads();
            // row r0 holds e0; rows k >= 1 start after it
            for (uint32_t k = threadIdx.x; k < rows; k += kPermThreads) {
                const uint64_t at = noff[r0 + k], end = noff[r0 + k + 1];
                s_shift[k] = static_cast<int64_t>(off[order[r0 + k]]) - static_cast<int64_t>(at);
                if (k && end > at && at - e0 < kTileEdges) s_row[at - e0] = static_cast<uint16_t>(k);
            }
            __syncthreads();
            // inclusive max-scan; thread i owns positions [8i, 8i + 8)
            const uint4 q = reinterpret_cast<const uint4 *>(s_row)[threadIdx.x];
            uint32_t v[8] = {q.x & 0xFFFFu, q.x >> 16, q.y & 0xFFFFu, q.y >> 16,
                             q.z & 0xFFFFu, q.z >> 16, q.w & 0xFFFFu, q.w >> 16};
#pragma unroll
            for (int j = 1; j < 8; ++j) v[j] = max(v[j], v[j - 1]);
            uint32_t run = v[7];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, run, o);
                if (lane >= o) run = max(run, y);
            }
            if (lane == 31) s_warp[warp] = run;
            uint32_t before = __shfl_up_sync(0xffffffffu, run, 1);
            if (lane == 0) before = 0;
            __syncthreads();
            for (int x = 0; x < warp; ++x) before = max(before, s_warp[x]);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = max(v[j], before);
            reinterpret_cast<uint4 *>(s_row)[threadIdx.x] = make_uint4(v[0] | (v[1] << 16), v[2] | (v[3] << 16),
                                                                       v[4] | (v[5] << 16), v[6] | (v[7] << 16));
            __syncthreads();
        }
        uint64_t src[kPermEdges];
#pragma unroll
        for (int i = 0; i < kPermEdges; ++i) {
            const uint64_t e = e0 + uint64_t(i) * kPermThreads + threadIdx.x;
            src[i] = 0;
            if (e < e1) {
                if (staged) {
                    src[i] = static_cast<uint64_t>(static_cast<int64_t>(e) + s_shift[s_row[i * kPermThreads + threadIdx.x]]);
                } else {
                    const uint64_t r = row_of(noff, V, e);
                    src[i] = off[order[r]] + (e - noff[r]);
                }
            }
        }
        uint32_t c[kPermEdges], wv[kPermEdges];
#pragma unroll
        for (int i = 0; i < kPermEdges; ++i) {
            const bool live = e0 + uint64_t(i) * kPermThreads + threadIdx.x < e1;
            c[i] = live ? ld_stream(cols + src[i]) : 0u;
            wv[i] = (live && w) ? ld_stream(w + src[i]) : 0u;
        }
        uint32_t nc[kPermEdges];
#pragma unroll
        for (int i = 0; i < kPermEdges; ++i) {
            const bool live = e0 + uint64_t(i) * kPermThreads + threadIdx.x < e1;
            nc[i] = 0;
            if (live && c[i] < V) {
                nc[i] = ld_nc_keep(inv + c[i], pol);
            } else if (live) {
                b |= kBadColumn;
            }
        }
#pragma unroll
        for (int i = 0; i < kPermEdges; ++i) {
            const uint64_t e = e0 + uint64_t(i) * kPermThreads + threadIdx.x;
            if (e < e1) {
                __stcs(ncols + e, nc[i]);
                if (nw) __stcs(nw + e, wv[i]);
            }
        }
        __syncthreads();  // the next tile overwrites the staged rows
    }
    if (b) atomicOr(bad, b);
}

// Graphs of up to this many vertices are ranked by one sort of all of them; leaving
// out those without a score first costs a selection and a read-back in mid-call.
constexpr uint64_t kWholeSort = 2048;

// Stable descending sort of (key, id) pairs on key bits [0, end_bit); the
// result ends in *keys / *ids (which may swap with the alternate buffers).
void sort_desc(uint64_t *&keys, uint64_t *keys_alt, uint32_t *&ids, uint32_t *ids_alt, uint64_t n, int end_bit,
               cudaStream_t s) {
    if (n < 2) return;
    cub::DoubleBuffer<uint64_t> kb(keys, keys_alt);
    cub::DoubleBuffer<uint32_t> vb(ids, ids_alt);
    size_t tb = 0;
    HYT_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tb, kb, vb, static_cast<int64_t>(n), 0, end_bit, s));
    Scratch<uint8_t> tmp(tb, s);
    HYT_CUDA(cub::DeviceRadixSort::SortPairsDescending(tmp.get(), tb, kb, vb, static_cast<int64_t>(n), 0, end_bit, s));
    keys = kb.Current();
    ids = vb.Current();
}

// out = indices i < n with flags[i] != 0, ascending (count to *count).
void select_index(const uint8_t *flags, uint32_t *out, uint64_t n, uint64_t *count, cudaStream_t s) {
    thrust::counting_iterator<uint32_t> it(0);
    size_t tb = 0;
    HYT_CUDA(cub::DeviceSelect::Flagged(nullptr, tb, it, flags, out, count, static_cast<int64_t>(n), s));
    Scratch<uint8_t> tmp(tb, s);
    HYT_CUDA(cub::DeviceSelect::Flagged(tmp.get(), tb, it, flags, out, count, static_cast<int64_t>(n), s));
}

void exclusive_scan(const uint64_t *in, uint64_t *out, uint64_t n, cudaStream_t s) {
    size_t tb = 0;
    HYT_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, in, out, static_cast<int64_t>(n), s));
    Scratch<uint8_t> tmp(tb, s);
    HYT_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), tb, in, out, static_cast<int64_t>(n), s));
}

// Hub count rule of the reference (its long-double arithmetic, on the host).
uint64_t hub_count_for(uint64_t V, double fraction) {
    const long double requested = static_cast<long double>(V) * static_cast<long double>(fraction);
    const long double rounded = std::round(requested);
    const long double pick = std::fabs(requested - rounded) < 1e-12L ? rounded : std::ceil(requested);
    const uint64_t n = pick <= 0.0L ? 0 : static_cast<uint64_t>(pick);
    return n < V ? n : V;
}

uint32_t read_flags(const uint32_t *bad, cudaStream_t s) {
    uint32_t h = 0;
    HYT_CUDA(cudaMemcpyAsync(&h, bad, 4, cudaMemcpyDeviceToHost, s));
    HYT_CUDA(cudaStreamSynchronize(s));
    return h;
}

void fail_on_csr_flags(uint32_t h) {
    if (h & kBadOffsets) fail(HYT_E_INVALID, "row offsets must start at 0 and be non-decreasing");
    if (h & kBadTerminal) fail(HYT_E_INVALID, "terminal row offset must equal the number of edges");
    if (h & kBadColumn) fail(HYT_E_INVALID, "column index contains an invalid destination vertex ID");
}

unsigned grid_sm(unsigned per_sm) { return static_cast<unsigned>(sm_count()) * per_sm; }

}  // namespace

void hub_sort(const hyt_csr &csr, double fraction, uint32_t *order_out, double *scores_out, uint64_t *hub_count,
              hyt_reorder_stats *stats) {
    const uint64_t V = csr.num_vertices, E = csr.num_edges;
    if (stats) std::memset(stats, 0, sizeof(*stats));
    if (!order_out && V) fail(HYT_E_INVALID, "vertex_order output is NULL");
    if (!std::isfinite(fraction) || fraction < 0.0 || fraction > 1.0)
        fail(HYT_E_INVALID, "HubSortOptions.hub_fraction must be finite and in [0, 1]");
    if (V > 0xFFFFFFFFull) fail(HYT_E_INVALID, "hub sorting takes graphs of < 2^32 vertices");
    if (hub_count) *hub_count = 0;
    if (V == 0) return;
    if (!csr.row_offsets || (E && !csr.column_indices)) fail(HYT_E_INVALID, "CSR arrays are NULL");
    StreamHold st;
    cudaStream_t s = st.s;
    EventTimer whole, main_k;
    whole.start(s);
    std::unique_ptr<Scratch<uint64_t>> off_h;
    std::unique_ptr<Scratch<uint32_t>> cols_h;
    const uint64_t *off = device_view(csr.row_offsets, V + 1, off_h, s);
    const uint32_t *cols = device_view(csr.column_indices, E, cols_h, s);
    Scratch<uint32_t> indeg(V, s), bad(1, s), ids(V, s), ids_alt(V, s);
    Scratch<uint64_t> outdeg(V, s), key(V, s), key_srt(V, s), key_alt(V, s), rest(1, s);
    Scratch<uint8_t> is_other(V, s);
    Scratch<unsigned long long> maxes(2, s);
    HYT_CUDA(cudaMemsetAsync(indeg.get(), 0, V * 4, s));
    HYT_CUDA(cudaMemsetAsync(bad.get(), 0, 4, s));
    HYT_CUDA(cudaMemsetAsync(maxes.get(), 0, 16, s));
    main_k.start(s);
    constexpr int kTable = 2 * kDegreeSlots * sizeof(uint32_t);
    HYT_CUDA(cudaFuncSetAttribute(degree_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTable));
    // no more CTAs than have a few edges per table slot (each clears and
    // flushes its table)
    const unsigned ctas = static_cast<unsigned>(
        std::min<uint64_t>(grid_sm(2), std::max<uint64_t>(1, std::max(E, V) / (2 * kDegreeThreads))));
    degree_pass_kernel<<<ctas, kDegreeThreads, kTable, s>>>(off, cols, V, E, indeg.get(), outdeg.get(), maxes.get(),
                                                            bad.get());
    main_k.stop(s);
    max_in_degree_kernel<<<grid_for(V, 256, 148u * 8u), 256, 0, s>>>(indeg.get(), V, maxes.get());
    const bool scores_dev = scores_out && is_device_pointer(scores_out);
    std::unique_ptr<Scratch<double>> sc;
    if (scores_out && !scores_dev) sc = std::make_unique<Scratch<double>>(V, s);
    double *scores_d = scores_dev ? scores_out : (sc ? sc->get() : nullptr);
    auto check_flags = [&] {  // waits for s
        const uint32_t h = read_flags(bad.get(), s);
        fail_on_csr_flags(h);
        if (h & kBadOverflow) fail(HYT_E_INVALID, "degree product exceeds 2^64");
    };
    const bool whole_sort = V <= kWholeSort;
    hub_scores_kernel<<<grid_sm(8), 256, 0, s>>>(outdeg.get(), indeg.get(), V, maxes.get(), scores_d, key.get(),
                                                 whole_sort ? nullptr : is_other.get(),
                                                 whole_sort ? ids.get() : nullptr, bad.get());
    HYT_CUDA(cudaGetLastError());
    if (scores_out && !scores_dev) HYT_CUDA(cudaMemcpyAsync(scores_out, scores_d, V * 8, cudaMemcpyDeviceToHost, s));
    // Only vertices with a score are ranked: the others tie at 0 and keep
    // their id order, which is where the stable sort would leave them too.  A
    // small graph is sorted whole, over the bits of any key.
    uint64_t scored = V;
    uint64_t *keys = key.get();
    uint32_t *ranked = ids.get();
    if (whole_sort) {
        sort_desc(keys, key_alt.get(), ranked, ids_alt.get(), V, 62, s);
    } else {
        select_index(is_other.get(), ids.get(), V, rest.get(), s);
        unsigned long long h_max[2] = {0, 0};
        HYT_CUDA(cudaMemcpyAsync(&scored, rest.get(), 8, cudaMemcpyDeviceToHost, s));
        HYT_CUDA(cudaMemcpyAsync(h_max, maxes.get(), 16, cudaMemcpyDeviceToHost, s));
        check_flags();
        const uint64_t denom = uint64_t(h_max[0]) * h_max[1];
        // products: the bits of the largest; scores in [0, 1]: 62 bits
        const int bits = denom < (uint64_t(1) << 52) ? (denom ? 64 - __builtin_clzll(denom) : 1) : 62;
        keys = key_srt.get();
        if (scored) {
            gather_keys_kernel<<<grid_for(scored, 256, 148u * 8u), 256, 0, s>>>(key.get(), ranked, scored, keys);
            HYT_CUDA(cudaGetLastError());
            sort_desc(keys, key_alt.get(), ranked, ids_alt.get(), scored, bits, s);
        }
    }
    const uint64_t hubs = hub_count_for(V, fraction);
    const uint64_t top = std::min(hubs, scored);
    // order = hubs (ranked; where the ranked run out, vertices of score 0 by
    // id), then the other vertices in id order: after the ranked hubs, all
    // the others in id order either way -- unless ranked ones are left over
    HYT_CUDA(cudaMemsetAsync(is_other.get(), 1, V, s));
    if (top) mark_kernel<<<grid_for(top, 256), 256, 0, s>>>(ranked, top, is_other.get());
    HYT_CUDA(cudaGetLastError());
    const bool order_dev = is_device_pointer(order_out);
    std::unique_ptr<Scratch<uint32_t>> ord;
    if (!order_dev) ord = std::make_unique<Scratch<uint32_t>>(V, s);
    uint32_t *order_d = order_dev ? order_out : ord->get();
    if (top) HYT_CUDA(cudaMemcpyAsync(order_d, ranked, top * 4, cudaMemcpyDeviceToDevice, s));
    select_index(is_other.get(), order_d + top, V, rest.get(), s);
    if (!order_dev) HYT_CUDA(cudaMemcpyAsync(order_out, order_d, V * 4, cudaMemcpyDeviceToHost, s));
    whole.stop(s);
    uint64_t h_rest = 0;
    HYT_CUDA(cudaMemcpyAsync(&h_rest, rest.get(), 8, cudaMemcpyDeviceToHost, s));
    if (whole_sort)
        check_flags();
    else
        HYT_CUDA(cudaStreamSynchronize(s));
    if (h_rest + top != V) fail(HYT_E_INTERNAL, "hub ordering lost vertices");
    if (hub_count) *hub_count = hubs;
    if (stats) {
        stats->device_ms = whole.ms();
        stats->kernel_ms = main_k.ms();
        stats->kernel_bytes = 4 * E + 16 * V;  // ids read; offsets read, out-degrees written
        // + in-degrees, scores / keys / ids written, the radix sort (12 B per
        // vertex read and written per 8-bit digit), the order and scores out
        stats->algorithmic_bytes = stats->kernel_bytes + 4 * V + 28 * V + 8 * 24 * V + 12 * V;
        stats->kernel_launches = hubs ? 4 : 3;
        stats->library_calls = 2;
    }
}

void csr_reorder(const hyt_csr &csr, const uint32_t *vertex_order, bool on_device, hyt_csr_buffers *out,
                 hyt_reorder_stats *stats, bool pooled) {
    const uint64_t V = csr.num_vertices, E = csr.num_edges;
    if (stats) std::memset(stats, 0, sizeof(*stats));
    if (!out || (!vertex_order && V)) fail(HYT_E_INVALID, "NULL argument");
    std::memset(out, 0, sizeof(*out));
    if (V > 0xFFFFFFFFull) fail(HYT_E_INVALID, "reordering takes graphs of < 2^32 vertices");
    if (csr.weight_kind != HYT_WEIGHTS_NONE && csr.weight_kind != HYT_WEIGHTS_F32 && csr.weight_kind != HYT_WEIGHTS_U32)
        fail(HYT_E_INVALID, "unknown weight kind");
    if (csr.weight_kind != HYT_WEIGHTS_NONE && E && !csr.weights) fail(HYT_E_INVALID, "weights are NULL");
    if (!csr.row_offsets || (E && !csr.column_indices)) fail(HYT_E_INVALID, "CSR arrays are NULL");
    const bool weighted = csr.weight_kind != HYT_WEIGHTS_NONE && E;
    StreamHold st;
    cudaStream_t s = st.s;
    EventTimer whole, main_k;
    whole.start(s);
    std::unique_ptr<Scratch<uint64_t>> off_h;
    std::unique_ptr<Scratch<uint32_t>> cols_h, w_h, order_h;
    const uint64_t *off = device_view(csr.row_offsets, V + 1, off_h, s);
    const uint32_t *cols = device_view(csr.column_indices, E, cols_h, s);
    const uint32_t *w = weighted ? device_view(static_cast<const uint32_t *>(csr.weights), E, w_h, s) : nullptr;
    const uint32_t *order = device_view(vertex_order, V, order_h, s);
    Scratch<uint32_t> inv(V, s), bad(1, s);
    Scratch<uint64_t> ndeg(V + 1, s);
    HYT_CUDA(cudaMemsetAsync(inv.get(), 0xFF, std::max<uint64_t>(V, 1) * 4, s));
    HYT_CUDA(cudaMemsetAsync(bad.get(), 0, 4, s));
    order_pass_kernel<<<grid_sm(8), 256, 0, s>>>(off, order, V, E, inv.get(), ndeg.get(), bad.get());
    HYT_CUDA(cudaGetLastError());
    // the permutation and the offsets must be valid before any kernel
    // indexes through them
    uint32_t h = read_flags(bad.get(), s);
    if (h & kBadOrderRange)
        fail(HYT_E_INVALID, "CSRGraph::reorder_vertices: vertex_order contains an out-of-range vertex ID");
    if (h & kBadOrderDup) fail(HYT_E_INVALID, "CSRGraph::reorder_vertices: vertex_order contains duplicate vertex IDs");
    fail_on_csr_flags(h);
    auto alloc = [&](size_t bytes) -> void * {
        void *p = nullptr;
        if (on_device && pooled) {
            int dev = 0;
            HYT_CUDA(cudaGetDevice(&dev));
            HYT_ALLOC(cudaMallocFromPoolAsync(&p, bytes ? bytes : 16, graph_pool(dev), cudaStreamLegacy));
            HYT_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
        } else if (on_device) {
            p = output_alloc(bytes);
        } else {
            p = std::malloc(bytes ? bytes : 16);
            if (!p) fail(HYT_E_OOM, "host allocation failed");
        }
        return p;
    };
    struct OutGuard {  // frees the outputs if a later step fails
        hyt_csr_buffers *o;
        bool pooled;
        bool armed = true;
        ~OutGuard() {
            if (!armed) return;
            if (pooled) {
                free_pooled_buffers(o);
            } else {
                hyt_csr_buffers_free(o);
            }
        }
    } guard{out, pooled && on_device};
    out->num_vertices = V;
    out->num_edges = E;
    out->on_device = on_device ? 1u : 0u;
    out->weight_kind = weighted ? csr.weight_kind : HYT_WEIGHTS_NONE;
    out->row_offsets = static_cast<uint64_t *>(alloc((V + 1) * 8));
    out->column_indices = static_cast<uint32_t *>(alloc(E * 4));
    if (weighted) out->weights = static_cast<uint32_t *>(alloc(E * 4));
    // host output: the kernels write device scratch, copied out at the end
    std::unique_ptr<Scratch<uint64_t>> noff_s;
    std::unique_ptr<Scratch<uint32_t>> ncols_s, nw_s;
    uint64_t *noff = out->row_offsets;
    uint32_t *ncols = out->column_indices, *nw = out->weights;
    if (!on_device) {
        noff_s = std::make_unique<Scratch<uint64_t>>(V + 1, s);
        ncols_s = std::make_unique<Scratch<uint32_t>>(E, s);
        noff = noff_s->get();
        ncols = ncols_s->get();
        if (weighted) {
            nw_s = std::make_unique<Scratch<uint32_t>>(E, s);
            nw = nw_s->get();
        }
    }
    exclusive_scan(ndeg.get(), noff, V + 1, s);
    const uint64_t tiles = (E + kTileEdges - 1) / kTileEdges;
    Scratch<uint64_t> tile_row(tiles + 1, s);
    if (E) tile_rows_kernel<<<grid_for(tiles + 1, 256), 256, 0, s>>>(noff, V, E, tiles, tile_row.get());
    main_k.start(s);
    if (E) {
        const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(tiles, grid_sm(5)));
        permute_edges_kernel<<<grid, kPermThreads, 0, s>>>(off, cols, w, noff, tile_row.get(), order, inv.get(), V, E,
                                                           ncols, weighted ? nw : nullptr, bad.get());
    }
    main_k.stop(s);
    HYT_CUDA(cudaGetLastError());
    if (!on_device) {
        HYT_CUDA(cudaMemcpyAsync(out->row_offsets, noff, (V + 1) * 8, cudaMemcpyDeviceToHost, s));
        if (E) HYT_CUDA(cudaMemcpyAsync(out->column_indices, ncols, E * 4, cudaMemcpyDeviceToHost, s));
        if (weighted) HYT_CUDA(cudaMemcpyAsync(out->weights, nw, E * 4, cudaMemcpyDeviceToHost, s));
    }
    whole.stop(s);
    h = read_flags(bad.get(), s);
    fail_on_csr_flags(h);
    guard.armed = false;
    if (stats) {
        stats->device_ms = whole.ms();
        stats->kernel_ms = main_k.ms();
        // ids read, renamed through inv and written; weights read and
        // written; per row a new start, an order entry and an old start
        stats->kernel_bytes = 12 * E + (weighted ? 8 * E : 0) + 20 * V;
        // + the order pass (order, offset pairs, inverse, degrees) and the scan
        stats->algorithmic_bytes = stats->kernel_bytes + 4 * V + 16 * V + 4 * V + 8 * V + 16 * V;
        stats->kernel_launches = E ? 3 : 1;
        stats->library_calls = 1;
    }
}

void free_pooled_buffers(hyt_csr_buffers *b) {
    if (!b) return;
    cudaDeviceSynchronize();
    for (void *p : {static_cast<void *>(b->row_offsets), static_cast<void *>(b->column_indices),
                    static_cast<void *>(b->weights)})
        if (p) cudaFreeAsync(p, cudaStreamLegacy);
    cudaStreamSynchronize(cudaStreamLegacy);
    std::memset(b, 0, sizeof(*b));
}

}  // namespace hyt
