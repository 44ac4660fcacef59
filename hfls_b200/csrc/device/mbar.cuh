// mbarrier helpers of the kernels whose warps or CTAs hand work to one
// another.  Every wait is bounded: TC_WAIT_LIMIT tries of up to
// TC_WAIT_HINT_NS each (a waiting thread is suspended until the phase
// completes or the hint runs out, so waiting warps leave the issue slots to
// the working ones); at most ~10 s in all before the wait reports a time-out.
#pragma once
#include <cstdint>

namespace htf {

constexpr unsigned TC_WAIT_LIMIT = 1u << 20;
constexpr unsigned TC_WAIT_HINT_NS = 10000;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes));
}

// returns false on time-out
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
    uint32_t done = 0;
    for (unsigned it = 0; it < TC_WAIT_LIMIT; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity), "r"(TC_WAIT_HINT_NS)
            : "memory");
        if (done) return true;
    }
    return false;
}

// one answer for all lanes of a warp: lanes try a barrier by themselves, so at the very limit one may give up on a
// phase that another still sees complete, and what follows (shuffles, matrix instructions, aligned barriers) wants
// the whole warp
__device__ __forceinline__ bool warp_agree(bool ok) { return __all_sync(0xffffffffu, ok); }

}  // namespace htf
