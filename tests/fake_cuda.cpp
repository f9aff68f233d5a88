// A host-only stand-in for the CUDA runtime calls of gg_copy.cu: copies happen at once, every
// handle remembers its device, and calls can be told to fail.
#include <cuda_runtime.h>

#include <atomic>
#include <cstring>

#include "gg_handle.h"

std::atomic<int> f_device{0}, f_registers{0}, f_unregisters{0}, f_copies{0}, f_syncs{0};
std::atomic<bool> f_refuse_register{false};
thread_local int t_device = 0;

struct FakeEvent { int device; };
struct FakeStream { int device; };

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void*, size_t, unsigned) {
    f_registers++;
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

namespace gg {
void* dev_alloc(size_t, int*) { return nullptr; }
void dev_free(void*, size_t, int) {}
}  // namespace gg
