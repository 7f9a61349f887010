// Programmatic dependent launches: a kernel queued behind another one in the
// same stream is set up (its CTAs placed, its parameters fetched) while the
// last CTAs of the one before still run, instead of after it has ended.
//
// Every kernel launched this way calls dependency_wait() before it touches
// memory that another kernel may write or still read: the call returns when all
// earlier grids of the stream have completed and their writes are visible, so
// the order of memory accesses is that of ordinary launches. That holds for
// ordinary loads only: a load through the read-only path (__ldg, or a const
// __restrict__ pointer) promises that nobody writes the memory while the kernel
// lives, and this kernel lives while the one before it writes. Only tables
// uploaded before the launches may be read that way.
// dependents_may_start() then lets the next grid be set up once every CTA of
// this one has got that far (all of them are resident by then, so a waiting
// grid never holds a place that a running one still needs).
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace emg {

__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace emg
