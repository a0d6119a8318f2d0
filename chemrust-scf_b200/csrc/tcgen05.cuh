// PTX helpers shared by the tcgen05 kernels: mbarriers with bounded waits and
// the commit of issued MMAs.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace chfsi {

// hard cap on polls of one wait, whatever the clock says
constexpr long long kSpinLimit = 1LL << 30;
// time limit of one wait in normal operation (a whole GEMM takes milliseconds)
constexpr unsigned long long kWaitNs = 4000000000ULL;
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

// Parity wait bounded by wait_ns of device time (and kSpinLimit polls);
// returns false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          unsigned long long wait_ns) {
    const uint32_t a = smem_u32(bar);
    const unsigned long long t0 = global_ns();
    for (long long i = 0; i < kSpinLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((i & 63) == 63 && global_ns() - t0 > wait_ns) return false;
    }
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// The same wait for kernels whose roles loop over many tiles: gives up as
// well once another role of the CTA has raised the abort flag.
__device__ __forceinline__ bool mbar_wait_or(uint64_t* bar, uint32_t parity,
                                             unsigned long long wait_ns,
                                             volatile const int* abort_flag) {
    const uint32_t a = smem_u32(bar);
    unsigned long long t0 = 0;  // the clock is read only once a wait is long
    for (long long i = 0; i < kSpinLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((i & 63) == 63) {
            if (*abort_flag) return false;
            const unsigned long long t = global_ns();
            if (t0 == 0) t0 = t;
            else if (t - t0 > wait_ns) return false;
        }
    }
    return false;
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(bar))
                 : "memory");
}

}  // namespace chfsi
