// Limit of a kernel's dynamic shared memory on the current device.
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace chfsi {

// Raises the limit to `bytes` where it is lower, and never lowers it: the
// attribute belongs to the kernel and the device, so another thread may be
// between its own call and its launch.
cudaError_t raise_smem_limit(const void* kernel, size_t bytes);
template <typename... A> cudaError_t raise_smem_limit(void (*kernel)(A...), size_t bytes) {
    return raise_smem_limit((const void*)kernel, bytes);
}

}  // namespace chfsi
