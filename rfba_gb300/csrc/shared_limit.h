// Dynamic shared memory of a launch.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace rfba {

// Lets kernel be launched with smem bytes of dynamic shared memory (a block has 227 KB
// with its static part). The limit belongs to the function, which contexts on other
// threads share, so it is set to the same value for every size: with the call's own
// size, another thread's smaller one could lower it between this and the launch.
template <class K>
cudaError_t allow_shared(K* kernel, size_t smem) {
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
    if (e != cudaSuccess) return e;
    const size_t limit = 227 * 1024 - a.sharedSizeBytes;
    if (smem > limit) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
}

}  // namespace rfba
