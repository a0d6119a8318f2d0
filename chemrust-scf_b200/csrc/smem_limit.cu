#include "smem_limit.hpp"

#include <mutex>
#include <unordered_map>

namespace chfsi {

namespace {
constexpr size_t kDefaultLimit = 48 * 1024;
std::mutex g_mu;
std::unordered_map<const void*, size_t> g_limit[64];
}  // namespace

cudaError_t raise_smem_limit(const void* kernel, size_t bytes) {
    if (bytes <= kDefaultLimit) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_mu);
    size_t& have = g_limit[dev][kernel];
    if (have >= bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) have = bytes;
    return e;
}

}  // namespace chfsi
