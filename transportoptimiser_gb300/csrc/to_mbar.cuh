// to_mbar.cuh - an mbarrier as a split CTA barrier: arrive when the own work
// is done, wait later.  Waits are bounded.
#pragma once
#include <cstdint>

namespace to_mbar {

__device__ __forceinline__ uint32_t addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// by one thread, before a CTA barrier
__device__ __forceinline__ void init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void arrive(uint64_t* bar) {
    asm volatile("{\n.reg .b64 s;\nmbarrier.arrive.shared::cta.b64 s, [%0];\n}"
                 :: "r"(addr(bar)) : "memory");
}
// until the phase of this parity has completed; false after 2^20 polls (each
// sleeps up to the hardware's own limit)
__device__ __forceinline__ bool wait(uint64_t* bar, uint32_t parity) {
    for (int it = 0; it < (1 << 20); ++it) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     "selp.b32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(addr(bar)), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}

}  // namespace to_mbar
