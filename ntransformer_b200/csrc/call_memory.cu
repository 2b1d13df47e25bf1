// call_memory.cu — memory that a call needs beside its arguments, in the order of its stream.
//
// CallMemory: from a pool of the call's device, so that calls on other streams, by other threads and on other devices have other memory, and a captured call has its
// graph's.  The pool keeps up to 64 MB between calls: the driver's own gives everything back whenever something waits for the stream and fetches it anew for the next call
// (a product of 16 tokens that is waited for: 455 us, 29 from this pool).
// StreamMemory: a buffer that the calls on one stream use in turn, for short calls, where taking memory and giving it back costs as much as the launches (decode
// attention that is waited for: 25.5 us, 23.1).  The lock is held until the call's last launch.
#include "kernels_internal.h"
#include <atomic>

namespace nt { namespace b200 {

namespace {

constexpr int DEVICES = 64, STREAMS = 16;
std::atomic<cudaMemPool_t> g_pool[DEVICES];

int device() {
    int dev = -1;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < DEVICES) return dev;
    cudaGetLastError();
    return -1;
}
cudaMemPool_t pool_of(int dev) {
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    cudaMemPool_t p = g_pool[dev].load();
    if (p) return p;
    // a first call may be under capture: making the pool is no part of it
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    const bool changed = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = CALL_MEMORY_KEPT;
    int off = 0;                                                   // no waits between streams for the sake of a block
    if (cudaMemPoolCreate(&p, &props) != cudaSuccess) p = nullptr;
    else if (cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
             cudaMemPoolSetAttribute(p, cudaMemPoolReuseAllowInternalDependencies, &off) != cudaSuccess) { cudaMemPoolDestroy(p); p = nullptr; }
    if (!p) cudaGetLastError();
    if (changed) cudaThreadExchangeStreamCaptureMode(&mode);
    g_pool[dev].store(p);
    return p;
}
void* take(size_t bytes, cudaStream_t s) {
    const int dev = device();
    if (dev < 0) return nullptr;
    cudaMemPool_t p = g_pool[dev].load();
    if (!p && !(p = pool_of(dev))) return nullptr;
    void* m = nullptr;
    if (cudaMallocFromPoolAsync(&m, bytes, p, s) != cudaSuccess) { cudaGetLastError(); return nullptr; }
    return m;
}

// Streams by the number that no other stream of the process has, then or later
struct Kept { int dev = -1; unsigned long long stream = 0; void* p = nullptr; size_t bytes = 0; };
Kept g_kept[STREAMS];
std::mutex g_kept_mu;

}  // namespace

CallMemory::CallMemory(size_t bytes, cudaStream_t s) : p(take(bytes, s)), stream(s) {}
CallMemory::~CallMemory() { if (p) NT_CUDA_CHECK(cudaFreeAsync(p, stream)); }

StreamMemory::StreamMemory(size_t bytes, cudaStream_t s) : stream(s) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamIsCapturing(s, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone && cudaStreamGetId(s, &id) == cudaSuccess) {
        lock = std::unique_lock<std::mutex>(g_kept_mu);
        Kept* k = nullptr;
        for (Kept& e : g_kept) if (e.p && e.stream == id) { k = &e; break; }
        if (k && k->bytes < bytes) {                               // behind the calls that use it
            NT_CUDA_CHECK(cudaFreeAsync(k->p, s));
            k->p = nullptr;
        }
        for (Kept& e : g_kept) if (!k && !e.p) k = &e;
        if (k && !k->p) {
            const size_t room = bytes < STREAM_MEMORY_LEAST ? STREAM_MEMORY_LEAST : bytes;
            if ((k->p = take(room, s))) { k->dev = device(); k->stream = id; k->bytes = room; }
        }
        if (k && k->p) { p = k->p; return; }
        lock.unlock();
    } else cudaGetLastError();
    p = take(bytes, s);                                            // captured, or more streams than are kept: the call's own
    own = p != nullptr;
}
StreamMemory::~StreamMemory() { if (own) NT_CUDA_CHECK(cudaFreeAsync(p, stream)); }

void trim_call_memory() {
    const int dev = device();
    if (dev < 0) return;
    {
        std::lock_guard<std::mutex> lk(g_kept_mu);
        bool any = false;
        for (const Kept& e : g_kept) any = any || (e.p && e.dev == dev);
        if (any && cudaDeviceSynchronize() == cudaSuccess)
            for (Kept& e : g_kept) if (e.p && e.dev == dev) { cudaFree(e.p); e = Kept(); }
    }
    if (cudaMemPool_t p = g_pool[dev].load()) cudaMemPoolTrimTo(p, 0);
    cudaGetLastError();
}

static std::atomic<int> g_users{0};
CallMemoryUser::CallMemoryUser() { g_users.fetch_add(1); }
CallMemoryUser::~CallMemoryUser() { if (g_users.fetch_sub(1) == 1) trim_call_memory(); }

}}  // namespace nt::b200

extern "C" void nt_b200_trim_memory(void) { nt::b200::trim_call_memory(); }
