// lg_launch.cuh -- kernel launches with a stated split between L1 and shared memory.
#pragma once
#include <cuda_runtime.h>

namespace lg {

// Launch with a share of the SM's memory set aside as shared memory (per cent; a hint). An SM changes that share
// only while it is idle, and by default it follows the kernel's own use.
template <typename... P, typename... A>
void launch_shared(int share, void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t st,
                   const A &...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    at.val.sharedMemCarveout = (unsigned)share;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace lg
