// Device arrays that a call hands to its caller (hyt_csr_buffers): cudaMalloc
// memory, as the interface says, so that a caller may export it to another
// process or map it for a peer.
//
// cudaMalloc and cudaFree of a renumbered graph cost more than the renumbering
// (0.5 GB on R-MAT scale 22: 3.2 ms a call against 0.8), so freed blocks are
// kept for the next call, up to kOutputKeep bytes and kOutputBlocks blocks per
// device, and returned when another allocation of this library finds no memory.  A
// free waits for the GPU first, as cudaFree does: the caller's own streams may
// still be reading, and the next owner writes.  (Blocks of the graph pool in their
// place could be handed on under such a reader, and could not be exported.)
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace hyt {

constexpr size_t kOutputKeep = size_t(4) << 30;  // a result of R-MAT scale 24 is 2.2 GiB: 10.3 ms a step without, 5.9 with
constexpr size_t kOutputBlocks = 64;  // small results: a block is searched for by size

// A cudaMalloc block of at least `bytes` on the current device.
void *output_alloc(size_t bytes);
// Frees a block that output_alloc(bytes) gave, or any other cudaMalloc memory.
void output_free(void *p, size_t bytes) noexcept;
// Returns a device's kept blocks to the driver; true when there were any.
bool output_release(int device) noexcept;

}  // namespace hyt
