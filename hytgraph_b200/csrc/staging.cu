// Copies between pageable host memory and the device through pinned chunks
// filled (or emptied) by several host threads; see staging.cuh.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "staging.cuh"

namespace hyt {
namespace {

constexpr size_t kChunk = size_t(1) << 20;      // per buffer
constexpr int kBuffers = 2;                     // per worker: one in flight, one being filled
constexpr int kMaxWorkers = 8;
// From these sizes on the threads, started on idle cores by each copy, save more than
// they cost.  Plain copy / through chunks, a pause before each copy as a solve makes
// one: to the device 2 MiB 0.23 / 0.24 ms, 4 MiB 0.41 / 0.29, 8 MiB 0.79 / 0.47, 128
// MiB 12.0 / 3.6; to the host 4 MiB 0.24 / 0.35, 8 MiB 0.43 / 0.61, 12 MiB 0.64 / 0.72,
// 16 MiB 0.83 / 0.74, 128 MiB 6.4 / 3.8, but into pages that nothing has touched yet
// 4 MiB 2.1 / 1.2, 8 MiB 4.1 / 1.7, 128 MiB 65 / 18.
constexpr size_t kMinBytes = size_t(4) << 20;
constexpr size_t kMinToTouched = size_t(16) << 20;

// True when most of the memory at p has no pages yet (a look at eight of them).
bool untouched(const void *p, size_t bytes) {
    const size_t page = static_cast<size_t>(sysconf(_SC_PAGESIZE));
    const uintptr_t first = reinterpret_cast<uintptr_t>(p) / page * page;
    int missing = 0;
    for (size_t k = 0; k < 8; ++k) {
        unsigned char resident = 1;
        const uintptr_t at = first + (2 * k + 1) * bytes / 16 / page * page;
        if (mincore(reinterpret_cast<void *>(at), page, &resident) == 0 && !(resident & 1)) ++missing;
    }
    return missing > 4;
}

// One worker's pinned buffers, stream and events on one device.
struct Lane {
    unsigned char *buf[kBuffers] = {};
    cudaStream_t stream = nullptr;
    cudaEvent_t done[kBuffers] = {};

    cudaError_t open() {
        cudaError_t e = cudaSuccess;
        for (int b = 0; b < kBuffers && e == cudaSuccess; ++b) {
            e = cudaHostAlloc(reinterpret_cast<void **>(&buf[b]), kChunk, cudaHostAllocPortable);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&done[b], cudaEventDisableTiming);
        }
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
        return e;
    }
    void close() {
        if (stream) cudaStreamSynchronize(stream), cudaStreamDestroy(stream);
        for (int b = 0; b < kBuffers; ++b) {
            if (done[b]) cudaEventDestroy(done[b]);
            if (buf[b]) cudaFreeHost(buf[b]);
        }
        *this = Lane{};
    }
};

struct Pool {
    std::mutex mu;  // one copy at a time per device
    std::vector<Lane> lanes;
    cudaEvent_t start = nullptr;
    bool failed = false;

    bool open() {
        if (failed) return false;
        if (!lanes.empty()) return true;
        const unsigned hw = std::thread::hardware_concurrency();
        lanes.resize(std::min<unsigned>(kMaxWorkers, std::max(1u, hw / 2)));
        cudaError_t e = cudaEventCreateWithFlags(&start, cudaEventDisableTiming);
        for (Lane &l : lanes)
            if (e == cudaSuccess) e = l.open();
        if (e == cudaSuccess) return true;
        (void)cudaGetLastError();
        close();
        failed = true;  // no pinned memory to be had: plain copies from now on
        return false;
    }
    void close() {
        for (Lane &l : lanes) l.close();
        lanes.clear();
        if (start) cudaEventDestroy(start);
        start = nullptr;
    }
};

std::mutex g_pools_mu;

Pool &pool_of(int device) {
    // never destroyed: at process exit the CUDA context may be gone first
    static auto *pools = new std::unordered_map<int, Pool>();
    std::lock_guard<std::mutex> lk(g_pools_mu);
    return (*pools)[device];
}

// Chunks `next`, `next` + 1, ... of the copy, taken one by one.
cudaError_t work(Lane &l, unsigned char *dst, const unsigned char *src, size_t bytes, bool to_device,
                 std::atomic<size_t> &next) {
    const cudaMemcpyKind kind = to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
    size_t off[kBuffers] = {}, len[kBuffers] = {};  // chunk in each buffer (len 0: none)
    cudaError_t e = cudaSuccess;
    auto settle = [&](int b) {
        if (!len[b]) return;
        const cudaError_t w = cudaEventSynchronize(l.done[b]);
        if (w == cudaSuccess && !to_device) std::memcpy(dst + off[b], l.buf[b], len[b]);
        if (e == cudaSuccess) e = w;
        len[b] = 0;
    };
    for (int b = 0; e == cudaSuccess; b = (b + 1) % kBuffers) {
        settle(b);
        const size_t at = next.fetch_add(1) * kChunk;
        if (at >= bytes || e != cudaSuccess) break;
        off[b] = at;
        len[b] = std::min(kChunk, bytes - at);
        if (to_device) {
            std::memcpy(l.buf[b], src + at, len[b]);
            e = cudaMemcpyAsync(dst + at, l.buf[b], len[b], kind, l.stream);
        } else {
            e = cudaMemcpyAsync(l.buf[b], src + at, len[b], kind, l.stream);
        }
        if (e == cudaSuccess) e = cudaEventRecord(l.done[b], l.stream);
        if (e != cudaSuccess) len[b] = 0;
    }
    for (int b = 0; b < kBuffers; ++b) settle(b);
    const cudaError_t w = cudaStreamSynchronize(l.stream);  // no copy may outlive its buffer's turn
    return e == cudaSuccess ? w : e;
}

}  // namespace

bool staged_copy(void *dst, const void *src, size_t bytes, bool to_device, cudaStream_t s) {
    if (bytes < kMinBytes) return false;
    if (!to_device && bytes < kMinToTouched && !untouched(dst, bytes)) return false;
    cudaPointerAttributes attr{};
    if (cudaPointerGetAttributes(&attr, to_device ? src : dst) != cudaSuccess) {
        (void)cudaGetLastError();
    } else if (attr.type != cudaMemoryTypeUnregistered) {
        return false;  // pinned (or device) memory copies at the link's speed by itself
    }
    int device = 0, of_stream = 0;
    HYT_CUDA(cudaGetDevice(&device));
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamGetDevice(s, &of_stream) != cudaSuccess || cudaStreamIsCapturing(s, &capture) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    if (of_stream != device) return false;  // the pool's events cannot be recorded on another device's stream
    if (capture != cudaStreamCaptureStatusNone) return false;  // its streams would join the capture
    Pool &p = pool_of(device);
    std::unique_lock<std::mutex> lk(p.mu, std::try_to_lock);
    if (!lk.owns_lock() || !p.open()) return false;
    // after everything queued on s; complete when this returns
    HYT_CUDA(cudaEventRecord(p.start, s));
    for (Lane &l : p.lanes) HYT_CUDA(cudaStreamWaitEvent(l.stream, p.start, 0));
    std::atomic<size_t> next{0};
    std::atomic<int> err{cudaSuccess};
    auto run = [&](Lane &l) {
        cudaError_t e = cudaSetDevice(device);
        if (e == cudaSuccess)
            e = work(l, static_cast<unsigned char *>(dst), static_cast<const unsigned char *>(src), bytes, to_device,
                     next);
        int none = cudaSuccess;
        if (e != cudaSuccess) err.compare_exchange_strong(none, e);
    };
    std::vector<std::thread> threads;
    const size_t workers = std::min(p.lanes.size(), (bytes + kChunk - 1) / kChunk);
    threads.reserve(workers);
    try {
        for (size_t i = 1; i < workers; ++i) threads.emplace_back([&run, &p, i] { run(p.lanes[i]); });
    } catch (const std::exception &) {  // fewer threads: the others take its chunks
    }
    run(p.lanes[0]);
    for (std::thread &t : threads) t.join();
    cuda_check(static_cast<cudaError_t>(err.load()), "copy through pinned chunks");
    return true;
}

void staging_release(int device) {
    Pool &p = pool_of(device);
    std::lock_guard<std::mutex> lk(p.mu);
    p.close();
    p.failed = false;
}

}  // namespace hyt
