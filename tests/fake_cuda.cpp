// A host-only stand-in for the CUDA runtime calls of gg_copy.cu and gg_alloc.cu: copies happen
// at once, events and streams remember their device, the device has as much memory as a test
// says, and calls can be told to fail.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>

std::atomic<int> f_device{0}, f_registers{0}, f_unregisters{0}, f_copies{0}, f_syncs{0};
std::atomic<bool> f_refuse_register{false};
thread_local int t_device = 0;

struct FakeEvent { int device; };
struct FakeStream { int device; };

// device memory: blocks of their true size, backed by 16 bytes
std::mutex f_mu;
std::map<void*, size_t> f_blocks;
size_t f_capacity = size_t(1) << 40, f_used = 0, f_registered = 0;

#undef cudaMalloc
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::mutex> lk(f_mu);
    if (f_used + n > f_capacity) return cudaErrorMemoryAllocation;
    *p = std::malloc(16);
    f_blocks[*p] = n;
    f_used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    std::lock_guard<std::mutex> lk(f_mu);
    f_used -= f_blocks.at(p);
    f_blocks.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void*, size_t n, unsigned) {
    f_registers++;
    f_registered = n;
    return f_refuse_register ? cudaErrorMemoryAllocation : cudaSuccess;
}
cudaError_t cudaHostUnregister(void*) { f_unregisters++; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(new FakeEvent{t_device});
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<FakeEvent*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    const bool same = reinterpret_cast<FakeEvent*>(e)->device == reinterpret_cast<FakeStream*>(s)->device;
    return same ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { f_syncs++; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t) {
    f_copies++;
    std::memcpy(to, from, n);
    return cudaSuccess;
}
}
