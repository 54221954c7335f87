// Programmatic dependent launch: chains of short kernels whose launch latency and prologue
// overlap the end of the kernel before.
//
// A kernel launched with launch_dependent() may start while its predecessor in the stream
// still runs. It calls dependent_prologue() before its first access to global memory: that
// lets its own successor start early and then waits until the predecessor has finished and
// its writes are visible. Every kernel of a chain waits, so the order of the whole chain
// holds. Before the call a kernel may only touch its parameters and shared memory. It reads
// global memory with coherent loads only: no __ldg, no ld.global.nc, no __restrict__ pointer. A
// read-only load wants data that nothing writes during the kernel's lifetime, which here begins
// while earlier kernels still write, and the compiler may move it above the wait.
// Measured on B200: a radix sort of 100,003 int64 keys (nine launches) 93 -> 70 us, of 2^20
// uint32 keys (five) 71 -> 60 us.
#pragma once

#include <cuda_runtime.h>

#include "runtime.hpp"

namespace pxb {

__device__ __forceinline__ void dependent_prologue() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

template <typename... P, typename... A>
inline bool launch_dependent(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                             cudaStream_t s, const char* what, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cuda_ok(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...), what);
}

}  // namespace pxb
