// mbarriers with bounded waits, and the Tensor Memory Accelerator's copies into this CTA's
// shared memory (no cluster multicast).
#pragma once

#include <cuda.h>

namespace opo {

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

constexpr long long kWaitCycles = 4000000000ll;  // ~2 s at 2 GHz
constexpr unsigned kWaitIters = 1u << 28;

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_test_wait(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Wait for the completion of the phase of parity `parity`; false when the bound
// (`cycles` SM clock cycles, or kWaitIters polls) expires.  try_wait may suspend the
// thread until the phase completes within a hardware time window, so a bound shorter
// than the default polls with the non-blocking test_wait instead: then the bound, not
// that window, ends the wait.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, long long cycles = kWaitCycles)
{
    const long long t0 = clock64();
    if (cycles < kWaitCycles) {
        for (unsigned it = 0; it < kWaitIters; it++) {
            if (mbar_test_wait(bar, parity)) return true;
            if (clock64() - t0 > cycles) break;
        }
        return false;
    }
    for (unsigned it = 0; it < kWaitIters; it++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (clock64() - t0 > cycles) break;
    }
    return false;
}

__device__ __forceinline__ void tma_tensor_3d(void *dst, const CUtensorMap *map, int c0, int c1, int c2,
                                              unsigned long long *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ void tma_bulk(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

}  // namespace opo
