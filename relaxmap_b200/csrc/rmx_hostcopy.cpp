#include "rmx_hostcopy.hpp"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

#include "rmx_common.cuh"
#include "rmx_io.hpp"

namespace rmx {
namespace {

constexpr int kThreads = 8, kSlots = 2 * kThreads;  // two slots per thread: one fills while the other is copied
constexpr size_t kSlotBytes = size_t(1) << 20;
// Below this a call does not allocate the ring (pinning its 16 MB takes about 7 ms once).
constexpr size_t kRingMin = size_t(32) << 20, kUseMin = size_t(4) << 20;

// One ring per process, used by one upload at a time (another copies as without it).
std::mutex g_ring_mu;
char *g_ring = nullptr;
int g_ring_dev = -1;  // device of the events
cudaEvent_t g_done[kSlots] = {};

void drop_ring() {
    if (!g_ring) return;
    int cur = -1;
    cudaGetDevice(&cur);
    if (cur != g_ring_dev) cudaSetDevice(g_ring_dev);
    for (cudaEvent_t &e : g_done) {
        if (e) {
            cudaEventSynchronize(e);
            cudaEventDestroy(e);
        }
        e = nullptr;
    }
    cudaFreeHost(g_ring);
    g_ring = nullptr;
    if (cur >= 0 && cur != g_ring_dev) cudaSetDevice(cur);
    (void)cudaGetLastError();
}

// The ring for device dev, or false (then the caller copies without it). The caller holds g_ring_mu.
bool ready_ring(int dev, size_t bytes) {
    if (g_ring && g_ring_dev == dev) return true;
    if (bytes < kRingMin) return false;
    drop_ring();
    g_ring_dev = dev;
    if (cudaHostAlloc(reinterpret_cast<void **>(&g_ring), kSlots * kSlotBytes, cudaHostAllocPortable) != cudaSuccess) {
        (void)cudaGetLastError();
        g_ring = nullptr;
        return false;
    }
    for (cudaEvent_t &e : g_done)
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            (void)cudaGetLastError();
            e = nullptr;
            drop_ring();
            return false;
        }
    return true;
}

bool is_pageable(const void *p) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return true;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

// Whether 16 of the array's pages, spread from its first to its last, are all in memory.
bool resident(const char *p, size_t bytes, size_t page) {
    constexpr size_t kSamples = 16;
    for (size_t k = 0; k < kSamples; k++) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p) + (bytes - 1) * k / (kSamples - 1);
        unsigned char in = 0;
        if (mincore(reinterpret_cast<void *>(a & ~(uintptr_t)(page - 1)), page, &in) != 0 || !(in & 1)) return false;
    }
    return true;
}

int host_threads(size_t bytes, size_t per_thread, size_t most) {
    const size_t hw = std::max(1u, std::thread::hardware_concurrency());
    return (int)std::max<size_t>(1, std::min({most, hw, bytes / per_thread}));
}

}  // namespace

void upload(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    if (bytes == 0) return;
    const int T = host_threads(bytes, kSlotBytes, kThreads);
    if (bytes >= kUseMin && T > 1 && is_pageable(src)) {
        std::unique_lock<std::mutex> lk(g_ring_mu, std::try_to_lock);
        int dev = 0;
        if (lk.owns_lock() && cudaGetDevice(&dev) == cudaSuccess && ready_ring(dev, bytes)) {
            const size_t n = (bytes + kSlotBytes - 1) / kSlotBytes;
            run_parallel(T, [&](int t) {  // thread t: chunks t, t + T, ... through its own two slots
                RMX_CUDA(cudaSetDevice(dev));
                int k = 0;
                for (size_t c = t; c < n; c += T, k ^= 1) {
                    const int slot = 2 * t + k;
                    const size_t off = c * kSlotBytes, len = std::min(kSlotBytes, bytes - off);
                    RMX_CUDA(cudaEventSynchronize(g_done[slot]));  // its last copy (of any call) is through
                    std::memcpy(g_ring + slot * kSlotBytes, static_cast<const char *>(src) + off, len);
                    RMX_CUDA(cudaMemcpyAsync(static_cast<char *>(dst) + off, g_ring + slot * kSlotBytes, len,
                                             cudaMemcpyHostToDevice, s));
                    RMX_CUDA(cudaEventRecord(g_done[slot], s));
                }
            });
            return;
        }
    }
    RMX_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
}

void download(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    if (bytes == 0) return;
    const int T = bytes < kUseMin ? 1 : host_threads(bytes, size_t(1) << 20, 16);
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    if (T > 1 && is_pageable(dst) && !resident(static_cast<const char *>(dst), bytes, page)) {
        const size_t pages = (bytes + page - 1) / page;
        char *const p = static_cast<char *>(dst);
        run_parallel(T, [&](int t) {  // a write that changes nothing maps the page
            for (size_t k = pages * t / T; k < pages * (t + 1) / T; k++) __atomic_fetch_or(p + k * page, 0, __ATOMIC_RELAXED);
        });
    }
    RMX_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
}

void release_upload_ring() {
    std::lock_guard<std::mutex> lk(g_ring_mu);
    drop_ring();
}

}  // namespace rmx
