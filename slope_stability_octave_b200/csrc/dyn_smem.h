// Opt-in to more than 48 KB of dynamic shared memory.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include <vector>

namespace sg {

// Raises the kernel's limit on the current device to `bytes`.  The limit belongs to the device, so
// what has been raised is remembered by (kernel, device); each host thread keeps its own list.
inline cudaError_t allow_dynamic_smem(const void *kernel, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    struct Raised {
        const void *kernel;
        int device;
        size_t bytes;
    };
    static thread_local std::vector<Raised> raised;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    Raised *at = nullptr;
    for (Raised &r : raised)
        if (r.kernel == kernel && r.device == device) at = &r;
    if (at && bytes <= at->bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    if (at) at->bytes = bytes;
    else raised.push_back({kernel, device, bytes});
    return cudaSuccess;
}

// the same for a kernel given by its name
template <typename... Args>
inline cudaError_t allow_dynamic_smem(void (*kernel)(Args...), size_t bytes) {
    return allow_dynamic_smem(reinterpret_cast<const void *>(kernel), bytes);
}

}  // namespace sg
