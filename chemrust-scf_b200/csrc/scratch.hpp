// Stream-ordered scratch of the entry points that take device pointers and
// have no context to keep buffers in (chfsi_zgemm_*, chfsi_hegv_dev).
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace chfsi {

// Freed scratch stays with the device up to this many bytes.
constexpr size_t kScratchKeep = (size_t)1 << 30;

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t st);
void scratch_free(void* p, cudaStream_t st);
// Gives the kept memory of all devices back: before an allocation is reported as
// failed, when the last context goes, and on chfsi_release_scratch.
void scratch_trim();
// cudaMalloc, with the kept scratch given back before it is refused.
cudaError_t malloc_or_trim(void** p, size_t bytes);

}  // namespace chfsi
