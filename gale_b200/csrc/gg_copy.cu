// gg_copy.cu -- host arrays to and from the device.
//
// The caller's arrays are pageable, and a cudaMemcpyAsync on pageable memory is staged by
// the driver on the calling thread: 170 MB of advected coordinates took 35 ms (5 GB/s,
// mostly page faults of the freshly allocated result), 28 MB of owning cells 1.6 ms, beside
// 1 ms and 0.5 ms of device work.  Transfers of kMinOut or kMinIn bytes and more are cut into
// chunks that kWorkers threads move through pinned slots: each thread copies its own chunks
// between the caller's memory and its two slots (the page faults then spread over the threads)
// while the copy engine moves the other slot, all on the handle's stream.  14 threads gained
// nothing (a transfer then waits for the last of them to wake).
//
// The slots (two per thread, pinned) and the threads are shared by the process, made once the
// transfers have earned them and given back when the last handle is destroyed.  One transfer
// uses them at a time; one that finds them busy (another thread's handle) takes the plain copy,
// so no caller waits for another.
//
// A program that keeps one handle at a time pays for the slots with each, so they have to
// be cheap: pinned pages of 4 KB cost 3.1 ms for 4 MB (cudaMallocHost) and 0.6 to give back, huge
// pages registered in place 0.55 and 0.25 (16 MB: 1.3-2.4 and 0.5).  And they have to be
// worth it: a handle that located 270 k points and was destroyed took 4.5 ms with 16 MB of slots
// made for its 1.1 MB of cells, 2.1 without.  The plain copy takes 0.22 µs per KB into fresh huge
// pages and 0.45 into small ones, staging 0.06, and on the way up it gains a quarter of that; so
// the bytes down and a quarter of the bytes up since no handle was alive are counted,
// kEarnSmall of them make slots of 256 KB (4 MB) and kEarnLarge slots of 1 MB (16 MB), which move
// 28 MB of cells in 1.3 ms instead of 1.8 and 170 MB of coordinates in 9.5 instead of 13.5
// (0.5 MB: 1.5 and 11.4; 2 MB: 1.3 and 10.4; device work included).
#include <emmintrin.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "gg_handle.h"
#include "gg_kernels.cuh"

namespace gg {

namespace {

constexpr int kWorkers = 8;
constexpr size_t kSlotSmall = size_t(256) << 10, kSlotLarge = size_t(1) << 20;
constexpr size_t kHugePage = size_t(2) << 20;
static_assert(kSlotSmall * 2 * kWorkers % kHugePage == 0, "the slots are whole huge pages");
constexpr size_t kMinChunk = size_t(128) << 10;
constexpr size_t kMinOut = size_t(1) << 20;   // to the host: the page faults alone pay for the threads
constexpr size_t kMinIn = size_t(12) << 20;   // to the device: the driver stages 3-10 MB as fast (0.34-1.06 ms), 21 MB in 2.2 ms against 1.7
// Results of this size go past the caches: through them their lines would lie, dirty, in the
// cores of the threads that wrote them, and the caller's thread would fetch them from there one
// by one (µs for a transfer into an array in use and a sum over it, plain copy / through the
// caches / past them: 4 MB 620 / 960 / 602, 8 MB 1220 / 1660 / 1160, 16 MB 2274 / 2180 / 2020).
// Smaller ones are with the caller's core soon enough (1.5 MB: 281 / 191 / 260), of larger ones the
// caches keep little (32 MB: 4544 / 3112 / 4160).
constexpr size_t kPastLo = size_t(7) << 18, kPastHi = size_t(18) << 20;
constexpr size_t kEarnSmall = size_t(8) << 20, kEarnLarge = size_t(128) << 20;

// memcpy past the caches
void stream_out(char* to, const char* from, size_t n) {
    const size_t head = std::min(n, (size_t)(-reinterpret_cast<uintptr_t>(to) & 15));
    std::memcpy(to, from, head);
    size_t i = head;
    for (; i + 64 <= n; i += 64) {
        __m128i v[4];
        for (int q = 0; q < 4; q++) v[q] = _mm_loadu_si128(reinterpret_cast<const __m128i*>(from + i + 16 * q));
        for (int q = 0; q < 4; q++) _mm_stream_si128(reinterpret_cast<__m128i*>(to + i + 16 * q), v[q]);
    }
    std::memcpy(to + i, from + i, n - i);
    _mm_sfence();
}

struct Job {
    char* host = nullptr;
    char* device = nullptr;
    size_t bytes = 0, chunk = 0;
    bool to_host = false;
    cudaStream_t stream = nullptr;
};

// The slots, their events and the threads of one device.
struct Stager {
    const int dev;
    const size_t slot;  // bytes of one of the 2·kWorkers slots
    const size_t all = slot * 2 * kWorkers;
    void* map = MAP_FAILED;  // the slots, with room to align them
    char* slots = nullptr;
    cudaEvent_t ev[kWorkers][2] = {};
    std::vector<std::thread> threads;
    std::mutex mu;
    std::condition_variable wake, idle;
    uint64_t generation = 0;
    int running = 0;
    bool stop = false;
    Job job;
    cudaError_t err = cudaSuccess;

    Stager(int d, size_t slot_bytes) : dev(d), slot(slot_bytes) {}

    bool start() {
        map = mmap(nullptr, all + kHugePage, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        if (map == MAP_FAILED) return false;
        const uintptr_t up = (reinterpret_cast<uintptr_t>(map) + kHugePage - 1) & ~(uintptr_t)(kHugePage - 1);
        slots = reinterpret_cast<char*>(up);
        madvise(slots, all, MADV_HUGEPAGE);  // refused: pages of 4 KB, which only cost time
        if (cudaHostRegister(slots, all, cudaHostRegisterPortable) != cudaSuccess) {
            cudaGetLastError();
            slots = nullptr;
            return false;
        }
        for (auto& e : ev)
            for (auto& x : e)
                if (cudaEventCreateWithFlags(&x, cudaEventDisableTiming) != cudaSuccess) {
                    cudaGetLastError();
                    return false;
                }
        try {
            for (int w = 1; w < kWorkers; w++) threads.emplace_back([this, w] { loop(w); });
        } catch (...) {
            return false;
        }
        return true;
    }

    ~Stager() {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop = true;
        }
        wake.notify_all();
        for (auto& t : threads) t.join();
        for (auto& e : ev)
            for (auto& x : e)
                if (x) cudaEventDestroy(x);
        if (slots) cudaHostUnregister(slots);
        if (map != MAP_FAILED) munmap(map, all + kHugePage);
    }

    void loop(int w) {
        cudaSetDevice(dev);
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lk(mu);
                wake.wait(lk, [&] { return stop || generation != seen; });
                if (stop) return;
                seen = generation;
            }
            const cudaError_t e = part(w);
            std::lock_guard<std::mutex> lk(mu);
            if (e != cudaSuccess && err == cudaSuccess) err = e;
            if (--running == 0) idle.notify_all();
        }
    }

    // this thread's chunks w, w + kWorkers, …
    cudaError_t part(int w) {
        const Job& j = job;
        const size_t n = (j.bytes + j.chunk - 1) / j.chunk;
        char* at[2] = {slots + (size_t)(2 * w) * slot, slots + (size_t)(2 * w + 1) * slot};
        auto size = [&](size_t k) { return std::min(j.chunk, j.bytes - k * j.chunk); };
        cudaError_t e = cudaSuccess;
        if (j.to_host) {
            const bool past_caches = j.bytes >= kPastLo && j.bytes < kPastHi;
            auto issue = [&](size_t k, int s) {
                e = cudaMemcpyAsync(at[s], j.device + k * j.chunk, size(k), cudaMemcpyDeviceToHost, j.stream);
                if (e == cudaSuccess) e = cudaEventRecord(ev[w][s], j.stream);
                return e == cudaSuccess;
            };
            int s = 0;
            bool ok = (size_t)w >= n || issue(w, 0);
            for (size_t k = w; k < n && ok; k += kWorkers, s ^= 1) {
                if (k + kWorkers < n) ok = issue(k + kWorkers, s ^ 1);
                const cudaError_t es = cudaEventSynchronize(ev[w][s]);
                if (e == cudaSuccess) e = es;
                ok = ok && es == cudaSuccess;
                if (ok && past_caches) stream_out(j.host + k * j.chunk, at[s], size(k));
                else if (ok) std::memcpy(j.host + k * j.chunk, at[s], size(k));
            }
        } else {
            int s = 0;
            bool used[2] = {false, false};
            for (size_t k = w; k < n && e == cudaSuccess; k += kWorkers, s ^= 1) {
                if (used[s]) e = cudaEventSynchronize(ev[w][s]);
                if (e != cudaSuccess) break;
                std::memcpy(at[s], j.host + k * j.chunk, size(k));
                e = cudaMemcpyAsync(j.device + k * j.chunk, at[s], size(k), cudaMemcpyHostToDevice, j.stream);
                if (e == cudaSuccess) e = cudaEventRecord(ev[w][s], j.stream);
                used[s] = true;
            }
            // the slots are free again only when their copies are done
            for (int q = 0; q < 2; q++)
                if (used[q]) {
                    const cudaError_t es = cudaEventSynchronize(ev[w][q]);
                    if (e == cudaSuccess) e = es;
                }
        }
        return e;
    }

    cudaError_t run(const Job& j) {
        {
            std::lock_guard<std::mutex> lk(mu);
            job = j;
            err = cudaSuccess;
            running = kWorkers - 1;
            generation++;
        }
        wake.notify_all();
        const cudaError_t e = part(0);
        std::unique_lock<std::mutex> lk(mu);
        idle.wait(lk, [&] { return running == 0; });
        const cudaError_t all = e != cudaSuccess ? e : err;
        if (all != cudaSuccess) cudaStreamSynchronize(j.stream);  // nothing may still use the slots
        return all;
    }
};

constexpr int kMaxDevices = 64;
struct PerDevice {
    std::mutex mu;  // held for the length of a staged transfer
    Stager* stager = nullptr;
    size_t earned = 0;     // bytes down and a quarter of the bytes up
    // slots could not be had (any, or larger ones): not tried again while handles live
    bool refused = false, keep_small = false;
};
// Never destroyed: threads may still wait on a stager when the process exits.
PerDevice& per_device(int dev) {
    static PerDevice* d = new PerDevice[kMaxDevices];
    return d[dev];
}
std::mutex g_handles_mu;
int g_handles = 0;
pid_t g_pid = 0;  // of the process whose handles these are

bool pageable(const void* host) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// false: not moved (small, pinned, busy or no slots, or the calling thread is on another
// device than the handle: its events could not be recorded on the handle's stream)
bool staged(Handle& H, void* host, void* device, size_t bytes, bool to_host) {
    if (bytes < (to_host ? kMinOut : kMinIn) || !pageable(host)) return false;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != H.device || dev < 0 || dev >= kMaxDevices) return false;
    PerDevice& D = per_device(dev);
    std::unique_lock<std::mutex> lk(D.mu, std::try_to_lock);
    if (!lk.owns_lock()) return false;
    if (D.refused) return false;
    D.earned += to_host ? bytes : bytes / 4;
    const size_t slot = D.earned >= kEarnLarge ? kSlotLarge : kSlotSmall;
    if (!D.stager && D.earned < kEarnSmall) return false;
    if (!D.stager || (D.stager->slot < slot && !D.keep_small)) {
        Stager* s = new (std::nothrow) Stager(dev, slot);
        if (s && s->start()) {
            delete D.stager;
            D.stager = s;
        } else {
            delete s;
            (D.stager ? D.keep_small : D.refused) = true;
            if (D.refused) return false;
        }
    }
    Job j;
    j.host = static_cast<char*>(host);
    j.device = static_cast<char*>(device);
    j.bytes = bytes;
    // every thread gets work, in chunks large enough to pay for their calls
    size_t c = (bytes / (2 * kWorkers) + 4095) & ~size_t(4095);
    j.chunk = c < kMinChunk ? kMinChunk : (c > D.stager->slot ? D.stager->slot : c);
    j.to_host = to_host;
    j.stream = H.stream;
    GG_CUDA(D.stager->run(j));
    return true;
}

}  // namespace

void copy_handle_created() {
    std::lock_guard<std::mutex> lk(g_handles_mu);
    if (g_handles++ == 0) g_pid = getpid();
}

void copy_handle_destroyed() {
    if (getpid() != g_pid) return;  // a child of fork: neither the threads nor CUDA came with it
    std::lock_guard<std::mutex> lk(g_handles_mu);
    if (--g_handles > 0) return;
    for (int dev = 0; dev < kMaxDevices; dev++) {
        PerDevice& D = per_device(dev);
        std::lock_guard<std::mutex> lk2(D.mu);
        delete D.stager;
        D.stager = nullptr;
        D.earned = 0;
        D.refused = D.keep_small = false;
    }
}

// Device → host after the stream's earlier work; the array is complete on return.
void copy_to_host(Handle& H, void* host, const void* device, size_t bytes) {
    if (staged(H, host, const_cast<void*>(device), bytes, true)) return;
    GG_CUDA(cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, H.stream));
    GG_CUDA(cudaStreamSynchronize(H.stream));
}

// Host → device, ordered before the stream's later work; the array may change on return.
void copy_to_device(Handle& H, void* device, const void* host, size_t bytes) {
    if (staged(H, const_cast<void*>(host), device, bytes, false)) return;
    GG_CUDA(cudaMemcpyAsync(device, host, bytes, cudaMemcpyHostToDevice, H.stream));
    if (!pageable(host)) GG_CUDA(cudaStreamSynchronize(H.stream));
}

}  // namespace gg
