// CPU tests of the pinned-chunk copies (hytgraph_b200/csrc/staging.cu) over a
// runtime made up here: two devices whose "memory" is host memory, and streams
// and events that know their device, as CUDA's do (an event recorded on a stream
// of another device is an invalid handle), and streams that a capture spreads to.
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "staging.cuh"

namespace {
struct Handle {
    int device;
    bool capturing = false;
};
thread_local int t_device = 0;
int copies = 0, failures = 0;
Handle g_legacy[2] = {{0}, {1}};

Handle *of(cudaStream_t s) { return s ? reinterpret_cast<Handle *>(s) : &g_legacy[t_device]; }
Handle *of(cudaEvent_t e) { return reinterpret_cast<Handle *>(e); }
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = t_device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return t_device = d, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidResourceHandle ? "invalid handle" : "error"; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return *p = std::malloc(n), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(new Handle{t_device}), cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
    return *e = reinterpret_cast<cudaEvent_t>(new Handle{t_device}), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return delete of(s), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete of(e), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    return of(s)->capturing ? cudaErrorStreamCaptureUnsupported : cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    return of(e)->capturing ? cudaErrorCapturedEvent : cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    if (of(e)->device != of(s)->device) return cudaErrorInvalidResourceHandle;
    return of(e)->capturing = of(s)->capturing, cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    if (of(e)->capturing) of(s)->capturing = true;  // joins the capture until that ends
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *c) {
    return *c = of(s)->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaStreamGetDevice(cudaStream_t s, int *d) { return *d = of(s)->device, cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    if (of(s)->capturing) return cudaSuccess;  // recorded, not run
    __atomic_add_fetch(&copies, 1, __ATOMIC_SEQ_CST);
    return std::memcpy(dst, src, n), cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
    std::memset(a, 0, sizeof(*a));
    return a->type = cudaMemoryTypeUnregistered, cudaSuccess;
}
// no device code in this program
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
char __cudaInitModule(void **) { return 0; }
}

namespace {
// What a copy of n bytes on `s` did: true when it went through the chunks and
// arrived; a copy that was left to the caller has touched nothing.
bool through_chunks(size_t n, bool to_device, cudaStream_t s, const char *what) {
    std::vector<unsigned char> src(n), dst(n, 0);
    for (size_t i = 0; i < n; ++i) src[i] = static_cast<unsigned char>(i * 7 + (i >> 13));
    copies = 0;
    try {
        const bool staged = hyt::staged_copy(dst.data(), src.data(), n, to_device, s);
        if (staged ? dst != src : copies != 0) {
            std::printf("FAILED %s: wrong bytes\n", what);
            ++failures;
        }
        return staged;
    } catch (const std::exception &e) {
        std::printf("FAILED %s: %s\n", what, e.what());
        ++failures;
        return false;
    }
}
void expect(bool got, bool want, const char *what) {
    if (got == want) return;
    std::printf("FAILED %s\n", what);
    ++failures;
}
}  // namespace

int main() {
    constexpr size_t kLarge = (size_t(33) << 20) + 12345;
    for (int current = 0; current < 2; ++current) {
        cudaSetDevice(current);
        cudaStream_t own = reinterpret_cast<cudaStream_t>(new Handle{current});
        cudaStream_t other = reinterpret_cast<cudaStream_t>(new Handle{1 - current});
        for (bool to_device : {true, false}) {
            expect(through_chunks(kLarge, to_device, own, "own stream"), true, "own stream");
            expect(through_chunks(kLarge, to_device, nullptr, "default stream"), true, "default stream");
            const size_t least = size_t(to_device ? 4 : 16) << 20;  // `dst` has its pages
            expect(through_chunks(least, to_device, own, "least copy"), true, "least copy");
            expect(through_chunks(least - 1, to_device, own, "small copy"), false, "small copy");
            // the runtime copies on a stream of any device: so must the caller, by itself
            expect(through_chunks(kLarge, to_device, other, "another device's stream"), false,
                   "another device's stream");
            // neither may a capture spread to the streams that all callers share
            Handle recording{current, true};
            expect(through_chunks(kLarge, to_device, reinterpret_cast<cudaStream_t>(&recording), "capturing stream"),
                   false, "capturing stream");
            expect(through_chunks(kLarge, to_device, own, "after a capturing stream"), true, "after a capturing stream");
            int d = -1;
            cudaGetDevice(&d);
            expect(d == current, true, "current device kept");
        }
    }
    // memory that nothing has touched yet is worth the chunks from 4 MiB on
    cudaSetDevice(0);
    for (size_t n : {size_t(4) << 20, (size_t(4) << 20) - 1, (size_t(9) << 20) + 12345}) {
        const std::vector<unsigned char> src(n, 5);
        void *m = mmap(nullptr, n + 8192, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        unsigned char *dst = static_cast<unsigned char *>(m) + 4099;
        const bool staged = hyt::staged_copy(dst, src.data(), n, false, nullptr);
        expect(staged, n >= size_t(4) << 20, "fresh memory");
        if (staged) expect(std::memcmp(dst, src.data(), n) == 0 && dst[-1] == 0 && dst[n] == 0, true, "fresh memory: bytes");
        munmap(m, n + 8192);
    }
    hyt::staging_release(0);
    hyt::staging_release(1);
    if (!failures) std::printf("staging tests passed\n");
    return failures ? 1 : 0;
}
