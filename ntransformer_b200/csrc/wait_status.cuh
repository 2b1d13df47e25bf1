// wait_status.cuh — waits for the phase of a copy, a product or a reader in the same CTA, with a limit.
//
// What is waited for is under way and takes microseconds.  Where it does not come within the limit the launch is broken: the wait says so in a status word
// that the host reads (kernels_internal.h wait_status).  Who was told so waits for nothing more and arrives on no barrier of the pipeline, so the others'
// waits run out as well; the loops go to their end (on whatever the stages hold: results are NaN or not written), and whoever issued copies or products
// waits for those in flight, again with a limit.
#pragma once
#include "ring.cuh"

namespace nt { namespace b200 {
namespace {

constexpr uint32_t WAIT_LIMIT_NS = 2000000000u;

__device__ __forceinline__ bool phase_done(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ uint32_t clock_ns() {
    uint32_t t;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
    return t;
}
__device__ __forceinline__ bool wait_phase(uint64_t* bar, uint32_t parity, unsigned* status, uint32_t limit_ns = WAIT_LIMIT_NS) {
    if (phase_done(bar, parity)) return true;
    const uint32_t t0 = clock_ns();
    while (!phase_done(bar, parity))
        if (clock_ns() - t0 > limit_ns) {
            if (status) asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(status), "r"(1u) : "memory");
            return false;
        }
    return true;
}
// In a loop whose instructions count: a lane that has once waited in vain (sound == false) goes on without waiting.
__device__ __forceinline__ void wait_sound(uint64_t* bar, uint32_t parity, unsigned* status, bool& sound) {
    if (phase_done(bar, parity) || !sound) return;
    sound = wait_phase(bar, parity, status);
}
// By a whole warp that leaves where the wait runs out: one answer for all lanes.
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, unsigned* status) { return __all_sync(0xFFFFFFFFu, wait_phase(bar, parity, status)) != 0; }

}  // namespace
}}  // namespace nt::b200
