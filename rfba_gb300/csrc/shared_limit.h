// Dynamic shared memory of a launch.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace rfba {

constexpr size_t kBlockShared = 227 * 1024;  // of a block, with its static part

// Lets kernel be launched with smem bytes of dynamic shared memory beside at most
// static_bytes of static. The limit belongs to the function, which contexts on other
// threads share, so it is set to the same value for every size: with the call's own
// size, another thread's smaller one could lower it between this and the launch.
template <class K>
cudaError_t allow_shared(K* kernel, size_t smem, size_t static_bytes) {
    const size_t limit = kBlockShared - static_bytes;
    if (smem > limit) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
}

// The same with the kernel's static part looked up (a few microseconds).
template <class K>
cudaError_t allow_shared(K* kernel, size_t smem) {
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
    return e != cudaSuccess ? e : allow_shared(kernel, smem, a.sharedSizeBytes);
}

}  // namespace rfba
