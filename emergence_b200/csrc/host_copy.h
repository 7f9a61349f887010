// Device → host copies into a caller's memory. A copy into pageable memory goes
// through one driver thread's staging buffer, which also takes the page faults of freshly allocated
// memory: 6-7 GB/s. Large ones therefore go through a library-owned pinned
// buffer that several host threads empty at once.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace emg {
// Queues the copy on `stream` and returns when the data is in `dst`.
cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream);
// Frees the pinned buffer, after the copy that may be using it (emg_release_memory).
void release_host_buffer();
}  // namespace emg
