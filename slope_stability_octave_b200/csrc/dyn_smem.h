// Opt-in to more than 48 KB of dynamic shared memory.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace sg {

// Raises the kernel's limit on the current device to `bytes`.  The limit belongs to the device, so
// what has been raised is remembered by (kernel, device); each host thread keeps its own list (a full
// list asks the driver each time).
inline cudaError_t allow_dynamic_smem(const void *kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    struct Raised {
        const void *kernel;
        int device;
        size_t bytes;
    };
    constexpr int most = 64;
    static thread_local Raised raised[most];
    static thread_local int count = 0;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    int at = 0;
    while (at < count && !(raised[at].kernel == kernel && raised[at].device == device)) ++at;
    if (at < count && bytes <= raised[at].bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess || at == most) return e;
    raised[at] = {kernel, device, bytes};
    if (at == count) ++count;
    return cudaSuccess;
}

// the same for a kernel given by its name
template <typename... Args>
inline cudaError_t allow_dynamic_smem(void (*kernel)(Args...), size_t bytes) {
    return allow_dynamic_smem(reinterpret_cast<const void *>(kernel), bytes);
}

}  // namespace sg
