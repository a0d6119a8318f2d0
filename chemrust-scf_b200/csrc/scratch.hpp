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
// Gives the kept memory of the current device back (before an allocation is
// reported as failed, and when the last context goes).
void scratch_trim();

}  // namespace chfsi
