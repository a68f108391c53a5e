// Pageable host memory <-> device copies at the host link's speed.
//
// The driver copies pageable memory through one pinned buffer with one thread: 11
// GB/s to the device, 20 back and 2 into pages that nothing has touched, on a host
// whose link takes 55.  Here up to 8 threads fill (or empty) 1 MiB pinned chunks and
// queue their copies on streams of their own: 35 GB/s up, 33 back, 7 into fresh
// pages; a job on 1 M vertices and 16 M edges from numpy arrays (upload, hub order,
// PageRank, one SSSP, results back) takes 9.6 ms in place of 19.1.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace hyt {

// Copies `bytes` between a host and a device address of the current device,
// after everything queued on s, and returns when they are there.  Returns
// false, with nothing copied, when a plain copy is as good (under 4 MiB, under 16
// MiB into host pages that are there already, pinned host memory, another thread's
// copy holds the chunks) or the only one that can follow s (a stream of another
// device, or one that is being captured).
bool staged_copy(void *dst, const void *src, size_t bytes, bool to_device, cudaStream_t s);

// Gives back a device's chunks (at most 16 MiB pinned), streams and events.
void staging_release(int device);

}  // namespace hyt
