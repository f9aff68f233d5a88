// gg_alloc.cu -- the device memory behind every handle buffer (DBuf).
//
// A handle sizes some 70 buffers on its first solve.  Through cudaMalloc those calls
// serialise in the driver: in a batch of 512 small problems driven by 64 host threads they
// took most of the wall time (36 k calls, 536 s summed over the threads, the batch at 53
// solves/s against 96 once every buffer existed).  Buffers of up to 4 MB therefore come from
// per-device pools: power-of-two size classes (256 B … 4 MB) carved from 64 MB chunks, with
// a free list per class, under one mutex per device.  Larger buffers (the fine-level
// moments, points and vectors of big meshes) still use cudaMalloc / cudaFree directly.
// Chunks stay with the process until it exits.
//
// An allocation that finds the device full takes back the scratch that handles of the same
// device keep between their calls (PointScratch) and tries once more.
//
// Reuse is as safe as with cudaFree, which synchronises the device: a block goes back on its
// free list only after cudaDeviceSynchronize, so no kernel of any stream still uses it when
// another handle is given it.
#include <algorithm>
#include <mutex>
#include <vector>

#include "gg_handle.h"

namespace gg {

namespace {

constexpr int kMinShift = 8;   // 256 B: every block keeps cudaMalloc's 256-byte alignment
constexpr int kMaxShift = 22;  // 4 MB
constexpr size_t kChunk = size_t(64) << 20;
constexpr int kMaxDevices = 64;

struct DevicePool {
    std::mutex mu;
    std::vector<void*> free_list[kMaxShift + 1];
    char* cur = nullptr;
    size_t left = 0;
};

// Never destroyed: a buffer released while the process exits still finds its pool.
DevicePool& pool(int dev) {
    static DevicePool* pools = new DevicePool[kMaxDevices];
    return pools[dev];
}

int size_class(size_t bytes) {
    int s = kMinShift;
    while ((size_t(1) << s) < bytes) s++;
    return s;
}

// Every handle's scratch.  Never destroyed, as the pools.
struct ScratchList {
    std::mutex mu;
    std::vector<PointScratch*> all;
};
ScratchList& scratch_list() {
    static ScratchList* l = new ScratchList;
    return *l;
}

// Give back the idle scratch on this device; a set in use (by this thread's own call too) stays.
bool reclaim_scratch(int dev) {
    ScratchList& L = scratch_list();
    std::lock_guard<std::mutex> lk(L.mu);
    bool any = false;
    for (PointScratch* s : L.all) {
        if (s->busy.exchange(true, std::memory_order_acquire)) continue;
        for (int k = 0; DBuf* b = s->all(k); k++)
            if (b->p && b->dev == dev) {
                b->release();
                any = true;
            }
        s->busy.store(false, std::memory_order_release);
    }
    return any;
}

void* device_malloc(size_t bytes, int dev) {
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation && reclaim_scratch(dev)) {
        cudaGetLastError();
        p = nullptr;
        e = cudaMalloc(&p, bytes);
    }
    GG_CUDA(e);
    return p;
}

}  // namespace

PointScratch::PointScratch() {
    ScratchList& L = scratch_list();
    std::lock_guard<std::mutex> lk(L.mu);
    L.all.push_back(this);
}

PointScratch::~PointScratch() {
    ScratchList& L = scratch_list();
    std::lock_guard<std::mutex> lk(L.mu);
    L.all.erase(std::find(L.all.begin(), L.all.end(), this));
}

void* dev_alloc(size_t bytes, int* dev_out) {
    int dev = 0;
    GG_CUDA(cudaGetDevice(&dev));
    *dev_out = dev;
    if (bytes > (size_t(1) << kMaxShift) || dev < 0 || dev >= kMaxDevices) return device_malloc(bytes, dev);
    const int s = size_class(bytes);
    const size_t sz = size_t(1) << s;
    DevicePool& P = pool(dev);
    for (bool retry = false;; retry = true) {
        {
            std::lock_guard<std::mutex> lk(P.mu);
            std::vector<void*>& fl = P.free_list[s];
            if (!fl.empty()) {
                void* p = fl.back();
                fl.pop_back();
                return p;
            }
            if (P.left < sz) {  // the rest of the current chunk (< 4 MB) is left unused
                void* c = nullptr;
                const cudaError_t e = cudaMalloc(&c, kChunk);
                if (e == cudaSuccess) {
                    P.cur = static_cast<char*>(c);
                    P.left = kChunk;
                } else if (retry || e != cudaErrorMemoryAllocation) {
                    GG_CUDA(e);
                } else {
                    cudaGetLastError();
                }
            }
            if (P.left >= sz) {
                void* p = P.cur;
                P.cur += sz;
                P.left -= sz;
                return p;
            }
        }
        reclaim_scratch(dev);  // without the lock: small scratch goes back to this pool
    }
}

void dev_free(void* p, size_t bytes, int dev) {
    if (!p) return;
    if (bytes > (size_t(1) << kMaxShift) || dev < 0 || dev >= kMaxDevices) {
        cudaFree(p);
        return;
    }
    int cur = 0;
    const bool switched = cudaGetDevice(&cur) == cudaSuccess && cur != dev;
    if (switched) cudaSetDevice(dev);
    cudaDeviceSynchronize();  // as cudaFree would: no stream of this device still uses p
    if (switched) cudaSetDevice(cur);
    DevicePool& P = pool(dev);
    std::lock_guard<std::mutex> lk(P.mu);
    P.free_list[size_class(bytes)].push_back(p);
}

}  // namespace gg
