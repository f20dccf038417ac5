// launch.cuh -- chained kernel launches.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace nxg {

uint32_t record_cuda(cudaError_t e);

namespace dev {

// Kernels of one call are chained as programmatic dependent launches: each
// lets the next one's CTAs be set up while it runs (chain_start) and touches
// memory only once the one before has completed and its writes are visible
// (chain_wait; a no-op in a kernel launched without the attribute).  That
// takes the launch gaps out of a chain of short kernels.
__device__ __forceinline__ void chain_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

} // namespace dev

// Launches `fn`; `chained`: as a programmatic dependent of the launch before it
// on the stream (fn then calls chain_wait before it touches memory).
template <class... Params, class... Args>
uint32_t launch_chained(bool chained, void (*fn)(Params...), uint32_t grid, uint32_t block, size_t shm,
                        cudaStream_t stream, const Args &...args) {
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(block);
    config.dynamicSmemBytes = shm;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = chained ? 1u : 0u;
    return record_cuda(cudaLaunchKernelEx(&config, fn, args...));
}

// Lets `fn` (of `fixed` bytes of static shared memory) be launched with any
// dynamic shared memory that a block may have, `optin` bytes in all.  The limit
// is the process's, so every call sets the same one: set to a call's own size,
// it could fall between another thread's setting and its launch.
inline uint32_t allow_shared(const void *fn, size_t fixed, int optin) {
    return record_cuda(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            optin - static_cast<int>(fixed)));
}

} // namespace nxg
