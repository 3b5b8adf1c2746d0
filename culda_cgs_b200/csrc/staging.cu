// staging.cu — large copies between pageable host memory and the device.
//
// The driver copies pageable memory through its own small pinned buffer on one
// thread: 122 MB of topics into a freshly allocated array took 26 to 34 ms (2.4
// ms on the link), 245 MB of doc ids on the way up 22 ms.  Here each of up to
// kSlots threads owns a pinned slot of one huge page's size and moves every
// kSlots-th block of the host array through it, so copying and the page faults
// of a new destination are spread over the threads while the link works on
// the other threads' slots: 5 ms each.  (A ring of 4 MB slots that all
// threads copied one after the other took 13 ms: two huge pages per slot give
// two of the threads all the faults.)
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <exception>
#include <mutex>
#include <new>
#include <thread>
#include <utility>

#include "internal.h"

namespace culda {

namespace {

constexpr size_t kSlotBytes = 2u << 20;
constexpr int kSlots = 8;
// Smaller arrays tend to lie in heap pages that are already mapped, into which the
// driver's copy runs at 16 to 18 GB/s: 10 MB take 0.56 ms, less than starting the
// threads adds.  At 24 MB a mapped destination takes 1.6 ms either way, a new
// one 6.2 ms by the driver's copy and 1.2 to 2 ms by this one.
constexpr size_t kStageMin = 16u << 20;

struct Ring {
    char *base = nullptr;              // kSlots slots of pinned memory
    cudaEvent_t free_at[kSlots] = {};  // the slot's last transfer
};

// Idle rings by device, at most kKept of each (release_staging frees them).
constexpr int kDevices = 64;
constexpr size_t kKept = 2;
std::mutex g_mu;
Ring *g_idle[kDevices][kKept] = {};

void free_ring(Ring *r) {
    for (cudaEvent_t e : r->free_at)
        if (e) {
            cudaEventSynchronize(e);
            cudaEventDestroy(e);
        }
    if (r->base) cudaFreeHost(r->base);
    delete r;
}

Ring *take_ring(int device) {
    {
        std::lock_guard<std::mutex> lock(g_mu);
        for (Ring *&kept : g_idle[device])
            if (kept) return std::exchange(kept, nullptr);
    }
    Ring *r = new (std::nothrow) Ring;
    if (!r) return nullptr;
    bool ok = cudaMallocHost((void **)&r->base, kSlotBytes * kSlots) == cudaSuccess;
    if (!ok) r->base = nullptr;
    for (cudaEvent_t &e : r->free_at)
        if (ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
            e = nullptr;
            ok = false;
        }
    if (!ok) {
        cudaGetLastError();
        free_ring(r);
        return nullptr;
    }
    return r;
}

void put_ring(int device, Ring *r) {
    {
        std::lock_guard<std::mutex> lock(g_mu);
        for (Ring *&kept : g_idle[device])
            if (!kept) {
                kept = r;
                return;
            }
    }
    free_ring(r);
}

// The ring for a copy of `bytes` at the host address p, or null when the copy
// should be a plain one (small, or not pageable memory).
Ring *ring_for(const void *p, size_t bytes, int &device) {
    if (bytes < kStageMin || cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kDevices) return nullptr;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return a.type == cudaMemoryTypeUnregistered ? take_ring(device) : nullptr;
}

}  // namespace

namespace {

// Moves `bytes` between the pageable host array and the device, block by block
// through the ring; blocks end on the host array's slot-size boundaries.
cudaError_t staged_copy(char *host, char *dev, size_t bytes, bool to_host, Ring *r, int device, cudaStream_t s) {
    const size_t head = reinterpret_cast<uintptr_t>(host) % kSlotBytes;  // before host in its first block
    const int64_t blocks = (int64_t)((head + bytes + kSlotBytes - 1) / kSlotBytes);
    std::atomic<int> failed{cudaSuccess};
    std::atomic<int64_t> next{0};
    // threads of this call only: nothing is left behind that a fork would break
    auto work = [&](int me) {
        char *slot = r->base + (size_t)me * kSlotBytes;
        cudaEvent_t moved = r->free_at[me];
        auto begin = [&](int64_t b) { return b == 0 ? 0 : (size_t)b * kSlotBytes - head; };
        auto size = [&](int64_t b) { return std::min((size_t)(b + 1) * kSlotBytes - head, bytes) - begin(b); };
        auto transfer = [&](int64_t b) {
            cudaError_t e = to_host ? cudaMemcpyAsync(slot, dev + begin(b), size(b), cudaMemcpyDeviceToHost, s)
                                    : cudaMemcpyAsync(dev + begin(b), slot, size(b), cudaMemcpyHostToDevice, s);
            return e == cudaSuccess ? cudaEventRecord(moved, s) : e;
        };
        cudaError_t e = cudaSetDevice(device);
        // the slot's last transfer, of an earlier copy
        if (e == cudaSuccess) e = cudaEventSynchronize(moved);
        int64_t b = next.fetch_add(1);
        if (to_host && e == cudaSuccess && b < blocks) e = transfer(b);
        while (b < blocks && e == cudaSuccess && failed.load() == cudaSuccess) {
            e = cudaEventSynchronize(moved);
            if (e != cudaSuccess) break;
            const int64_t after = next.fetch_add(1);
            if (to_host) {
                std::memcpy(host + begin(b), slot, size(b));
                if (after < blocks) e = transfer(after);
            } else {
                std::memcpy(slot, host + begin(b), size(b));
                e = transfer(b);
            }
            b = after;
        }
        if (e != cudaSuccess) failed.store(e);
    };
    std::thread team[kSlots];
    const int threads = (int)std::min<int64_t>(kSlots, blocks);
    try {
        for (int t = 1; t < threads; ++t) team[t] = std::thread(work, t);
    } catch (const std::exception &) {  // no more threads (or no memory for one): those that run share the blocks
    }
    work(0);
    for (std::thread &t : team)
        if (t.joinable()) t.join();
    const cudaError_t e = (cudaError_t)failed.load();
    if (e != cudaSuccess) cudaStreamSynchronize(s);  // nothing uses the ring any more
    return e;
}

}  // namespace

cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    int device = 0;
    if (Ring *r = ring_for(dst, bytes, device)) {
        const cudaError_t e =
            staged_copy(static_cast<char *>(dst), static_cast<char *>(const_cast<void *>(src)), bytes, true, r, device, s);
        put_ring(device, r);
        return e;
    }
    const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s);
    return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
}

cudaError_t copy_to_device(void *dst, const void *src, size_t bytes, cudaStream_t s) {
    int device = 0;
    Ring *r = ring_for(src, bytes, device);
    if (!r) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s);
    const cudaError_t e =
        staged_copy(static_cast<char *>(const_cast<void *>(src)), static_cast<char *>(dst), bytes, false, r, device, s);
    put_ring(device, r);  // the next user waits for a slot's transfer before it touches it
    return e;
}

void release_staging(int device) {
    if (device < 0 || device >= kDevices) return;
    Ring *idle[kKept];
    {
        std::lock_guard<std::mutex> lock(g_mu);
        for (size_t i = 0; i < kKept; ++i) idle[i] = std::exchange(g_idle[device][i], nullptr);
    }
    for (Ring *r : idle)
        if (r) free_ring(r);
}

}  // namespace culda
