// Kept cudaMalloc blocks of caller-owned results; see outputs.cuh.
#include <cuda.h>

#include <algorithm>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "outputs.cuh"

namespace hyt {
namespace {

struct Live {
    int device;
    size_t size, asked;  // of the block; by the caller it was handed to
};
struct Kept {
    int device;
    size_t size;
    void *p;
};
struct Blocks {
    std::mutex mu;
    std::unordered_map<void *, Live> live;
    std::vector<Kept> kept;  // oldest first
};

Blocks &blocks() {
    static auto *b = new Blocks();  // never destroyed: the CUDA context may be gone before it
    return *b;
}

// Waits for the work of every device in use (a peer may be reading too).
bool wait_for_devices() {
    static const auto state = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found{};
        if (cudaGetDriverEntryPoint("cuDevicePrimaryCtxGetState", &f, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<CUresult (*)(CUdevice, unsigned *, int *)>(f);
    }();
    int n = 0, cur = 0;
    if (cudaGetDevice(&cur) != cudaSuccess || cudaGetDeviceCount(&n) != cudaSuccess) return false;
    bool ok = cudaDeviceSynchronize() == cudaSuccess;
    for (int d = 0; d < n && ok; ++d) {
        unsigned flags = 0;
        int active = 0;
        if (d == cur) continue;
        if (!state || state(d, &flags, &active) != CUDA_SUCCESS) return false;
        if (active) ok = cudaSetDevice(d) == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
    }
    if (n > 1) cudaSetDevice(cur);
    return ok;
}

}  // namespace

void *output_alloc(size_t bytes) {
    Blocks &b = blocks();
    int device = 0;
    HYT_CUDA(cudaGetDevice(&device));
    std::unique_lock<std::mutex> lk(b.mu);
    // the smallest kept block that is large enough and wastes at most a quarter
    auto best = b.kept.end();
    for (auto k = b.kept.begin(); k != b.kept.end(); ++k)
        if (k->device == device && k->size >= bytes && k->size - bytes <= bytes / 4 &&
            (best == b.kept.end() || k->size < best->size))
            best = k;
    if (best != b.kept.end()) {
        void *p = best->p;
        b.live[p] = Live{device, best->size, bytes};
        b.kept.erase(best);
        return p;
    }
    void *p = nullptr;
    lk.unlock();
    HYT_ALLOC(cudaMalloc(&p, bytes ? bytes : 16));
    lk.lock();
    try {
        b.live[p] = Live{device, bytes ? bytes : 16, bytes};
    } catch (...) {
        cudaFree(p);
        throw;
    }
    return p;
}

void output_free(void *p, size_t bytes) noexcept {
    if (!p) return;
    Blocks &b = blocks();
    Live l{};
    {
        std::lock_guard<std::mutex> lk(b.mu);
        const auto it = b.live.find(p);
        if (it != b.live.end()) {
            // a block freed behind our back may have come back from cudaMalloc
            // at another size: only one that matches is known to be ours
            if (it->second.asked == bytes) l = it->second;
            b.live.erase(it);
        }
    }
    if (l.size == 0 || l.size > kOutputKeep || !wait_for_devices()) {
        cudaFree(p);
        return;
    }
    std::lock_guard<std::mutex> lk(b.mu);
    try {
        b.kept.push_back(Kept{l.device, l.size, p});
    } catch (...) {
        cudaFree(p);
        return;
    }
    size_t held = 0, count = 0;
    for (const Kept &k : b.kept)
        if (k.device == l.device) held += k.size, ++count;
    for (auto k = b.kept.begin(); held > kOutputKeep || count > kOutputBlocks;) {
        if (k->device != l.device) {
            ++k;
            continue;
        }
        held -= k->size;
        --count;
        cudaFree(k->p);
        k = b.kept.erase(k);
    }
}

bool output_release(int device) noexcept {
    Blocks &b = blocks();
    std::lock_guard<std::mutex> lk(b.mu);
    bool any = false;
    for (auto k = b.kept.begin(); k != b.kept.end();) {
        if (k->device != device) {
            ++k;
            continue;
        }
        cudaFree(k->p);
        k = b.kept.erase(k);
        any = true;
    }
    return any;
}

bool reclaim_device_memory(cudaError_t e) {
    if (e != cudaErrorMemoryAllocation) return false;
    (void)cudaGetLastError();
    int device = 0;
    return cudaGetDevice(&device) == cudaSuccess && output_release(device);
}

}  // namespace hyt
