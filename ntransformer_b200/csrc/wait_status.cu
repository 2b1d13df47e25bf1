// wait_status.cu — the status word of wait_status.cuh: one for the process, in pinned host memory that every device sees, so that reading it costs no copy.
#include "kernels_internal.h"
#include "wait_status.cuh"
#include "../../include/nt_b200.h"

namespace nt { namespace b200 {

namespace {

struct Word {
    volatile unsigned* host = nullptr;
    unsigned own = 0;                    // without a device: nothing writes, the host side works all the same
    Word() {
        // a first launch may be under capture: allocating is no part of it
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        const bool changed = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
        void* p = nullptr;
        if (cudaHostAlloc(&p, sizeof(unsigned), cudaHostAllocMapped | cudaHostAllocPortable) == cudaSuccess) host = static_cast<unsigned*>(p);
        else { cudaGetLastError(); host = &own; }
        if (changed) cudaThreadExchangeStreamCaptureMode(&mode);
        *host = 0;
    }
};
Word& word() { static Word w; return w; }

// waits for a phase that nothing completes
__global__ void wait_probe_kernel(unsigned* status, unsigned tries, int* came) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) { mbar_init(&bar, 1); mbar_fence_init(); }
    __syncthreads();
    wait_phase(&bar, 0, status, tries);
    if (threadIdx.x == 0) *came = tries != 0;
}
// lets the next launch start, and writes only then
__global__ void __launch_bounds__(1024) late_copy_kernel(uint32_t* dst, const uint32_t* src, size_t words, unsigned nanoseconds) {
    pdl_launch_dependents();
    pdl_wait();
    for (unsigned t = 0; t < nanoseconds; t += 1000) __nanosleep(1000);
    for (size_t i = threadIdx.x; i < words; i += 1024) dst[i] = src[i];
}

}  // namespace

unsigned* wait_status() { Word& w = word(); return w.host == &w.own ? nullptr : const_cast<unsigned*>(w.host); }
bool wait_expired() { return *word().host != 0; }

}}  // namespace nt::b200

extern "C" {
int nt_b200_wait_status(int set) {
    volatile unsigned* w = nt::b200::word().host;
    const int was = (int)*w;
    if (set >= 0) *w = (unsigned)set;
    return was;
}
void nt_b200_late_copy(void* dst, const void* src, size_t bytes, unsigned nanoseconds, void* stream) {
    nt::b200::launch_k_pdl(true, nt::b200::late_copy_kernel, dim3(1), dim3(1024), 0, static_cast<cudaStream_t>(stream), static_cast<uint32_t*>(dst), static_cast<const uint32_t*>(src),
                           bytes / 4, nanoseconds);
    nt::b200::count_launch();
}
void nt_b200_wait_probe(unsigned tries, int* came_dev, void* stream) {
    nt::b200::wait_probe_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(nt::b200::wait_status(), tries, came_dev);
    nt::b200::count_launch();
}
}
