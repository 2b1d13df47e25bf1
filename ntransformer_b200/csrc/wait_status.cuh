// wait_status.cuh — waits for the phase of a copy, a product or a reader in the same CTA, with a limit.
//
// What is waited for is under way and takes microseconds.  Where it does not come within the limit the launch is broken: the wait says so in a status word
// that the host reads (kernels_internal.h wait_status).  Who was told so waits for nothing more, the loops go to their end on whatever the stages hold, results
// are NaN or not written, and whoever issued copies or products waits for those in flight, again with a limit.
#pragma once
#include "ring.cuh"

namespace nt { namespace b200 {
namespace {

constexpr uint32_t WAIT_TRIES = 1u << 19;      // a try that fails suspends the thread for 4 us: 2 s

__device__ __forceinline__ bool phase_done(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return done != 0;
}
// tries: how often this lane still asks, WAIT_TRIES until a wait has run out and 0 from then on.
__device__ __forceinline__ void wait_phase(uint64_t* bar, uint32_t parity, unsigned* status, uint32_t& tries) {
    for (uint32_t i = 0; !phase_done(bar, parity); i++)
        if (i >= tries) {
            if (tries && status) asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(status), "r"(1u) : "memory");
            tries = 0;
            return;
        }
}
// The same without a register or an answer where either costs (the block GEMV's loops, a vote of the producer's warp included: 70B decode step 755 -> 765 us): a
// word at a fixed place in shared memory, zero at first, is set instead, and a wait that finds it set ends.
__device__ __forceinline__ bool word_set(uint32_t smem_addr) {
    uint32_t v;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_addr) : "memory");
    return v != 0;
}
__device__ __forceinline__ void set_word(uint32_t smem_addr, uint32_t v) { asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(smem_addr), "r"(v) : "memory"); }
__device__ __forceinline__ void wait_cta(uint64_t* bar, uint32_t parity, uint32_t dead) {
    asm volatile(
        "{\n"
        " .reg .pred p;\n"
        " .reg .b32 i, d;\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1;\n"
        " @p bra NT_CAME_%=;\n"
        " mov.b32 i, 0;\n"
        "NT_AGAIN_%=:\n"
        " mbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1;\n"
        " @p bra NT_CAME_%=;\n"
        " ld.volatile.shared.b32 d, [%2];\n"
        " setp.ne.b32 p, d, 0;\n"
        " @p bra NT_CAME_%=;\n"
        " add.u32 i, i, 1;\n"
        " setp.lt.u32 p, i, %3;\n"
        " @p bra NT_AGAIN_%=;\n"
        " st.volatile.shared.b32 [%2], i;\n"
        "NT_CAME_%=:\n"
        "}\n" ::"r"(smem_u32(bar)), "r"(parity), "r"(dead), "n"(WAIT_TRIES) : "memory");
}
__device__ __forceinline__ void report(unsigned* status) { if (status) asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(status), "r"(1u) : "memory"); }
// By a whole warp that leaves where the wait runs out: one answer for all lanes.
__device__ __forceinline__ bool wait_warp(uint64_t* bar, uint32_t parity, unsigned* status) {
    uint32_t tries = WAIT_TRIES;
    wait_phase(bar, parity, status, tries);
    return __all_sync(0xFFFFFFFFu, tries != 0) != 0;
}
// The last wait of a launch that is given up, for what it has in flight.
__device__ __forceinline__ void wait_flight(uint64_t* bar, uint32_t parity) {
    uint32_t tries = WAIT_TRIES;
    wait_phase(bar, parity, nullptr, tries);
}

}  // namespace
}}  // namespace nt::b200
