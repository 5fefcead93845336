// dev_pool.h -- the device memory of the handles.
//
// A handle's buffers (for a 720p grid 14, some 900 MB with its tables) are mapped when it is made and unmapped
// when it goes: more than the work of the calls that make a handle for one pass (the periodicity of one 720p
// frame: 4.5 of 7.5 ms). So what a handle gives back stays mapped for the next one, at most 1 GiB a device:
//
//   up to kPoolBuffer bytes   a CUDA memory pool of the library's own
//   above                     buffers from cudaMalloc, of which kLargeKeep bytes are kept, the last released
//
// What the pool has unused and the large buffers kept are kKeep bytes at most together; where they would be more, what was
// used last stays: a release of small buffers drops the oldest of the kept, one that keeps a large buffer what the
// pool has too much (balance).
//
// The line lies where the pool stops being the faster to map: new buffers of 1, 32, 64, 128 and 512 MiB take 0.23, 0.22,
// 0.41, 0.81 and 3.2 ms from the pool, which maps 2 MiB at a time, and 0.36, 0.34, 0.34, 0.35 and 0.58 ms from cudaMalloc; their
// release 0.20, 0.20, 0.40, 0.80 and 3.2 ms, and 0.30, 0.29, 0.30, 0.33 and 0.72 ms. Buffers that do not fit what is
// kept (the spectra of a dense 1080p grid, 0.6 GB and more each) are mapped for every handle, as by cudaMalloc alone; a
// large buffer is given out again only for one of its size or up to a fifth smaller, so handles of different
// geometries that come and go in turn map again what 1 GiB does not hold for both (1 to 2 ms a change).
// When the device is out of memory an allocation first returns all that is kept; release_memory() does so for others.
//
// The buffers are ready for, and freed after, every stream, as with cudaMalloc and cudaFree: an allocation
// waits for its (empty) stream, a release first for the device (wait_for_device). The contents of a buffer are
// undefined. Any thread may call, with any device current.
#pragma once

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <new>
#include <unordered_map>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

namespace b200 {

constexpr size_t kKeep = size_t(1) << 30;
constexpr size_t kLargeKeep = size_t(896) << 20;
constexpr size_t kPoolBuffer = size_t(32) << 20;
constexpr size_t kWaitBuffer = 256;

struct DevPool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;   // orders the pool's allocations and releases; no work runs on it
    void *anchor = nullptr;          // keeps a block of small buffers mapped for wait_for_device
    std::mutex mutex;                // of what follows
    std::unordered_map<void *, size_t> held;            // large buffers in use, with their sizes
    std::vector<std::pair<void *, size_t>> kept;        // and those kept, the oldest first
    size_t kept_bytes = 0;

    // The bound, after releases: of small buffers alone, or with large ones kept. (The pool's own threshold is no use for
    // it: it counts the buffers in use, and a few handles alive would have every release unmap memory.)
    void balance(bool large)
    {
        cudaStreamSynchronize(stream);   // the releases on it are then done
        uint64_t used = 0, reserved = 0;
        if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess ||
            cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        const size_t idle = reserved > used ? size_t(reserved - used) : 0;
        std::vector<std::pair<void *, size_t>> gone;
        size_t share = 0;
        {
            std::lock_guard<std::mutex> lock(mutex);
            if (!large) drop(idle < kKeep ? kKeep - idle : 0, gone);
            share = kKeep - kept_bytes;
        }
        for (auto &b : gone) cudaFree(b.first);
        if (idle > share) cudaMemPoolTrimTo(pool, size_t(used) + share);
    }
    // the oldest of the kept into gone, down to `most` bytes; under the lock
    void drop(size_t most, std::vector<std::pair<void *, size_t>> &gone)
    {
        size_t n = 0;
        while (kept_bytes > most) kept_bytes -= kept[n++].second;
        gone.insert(gone.end(), kept.begin(), kept.begin() + n);
        kept.erase(kept.begin(), kept.begin() + n);
    }
};

// the current device's pool (nullptr: it has none)
inline cudaError_t device_pool(DevPool *&out)
{
    static std::mutex mutex;
    static DevPool *pools[64] = {};   // outlive every handle
    static bool tried[64] = {};
    out = nullptr;
    int dev = 0;
    if (cudaError_t e = cudaGetDevice(&dev)) return e;
    if (dev < 0 || dev >= 64) return cudaSuccess;
    std::lock_guard<std::mutex> lock(mutex);
    if (!tried[dev]) {
        int has = 0;
        if (cudaDeviceGetAttribute(&has, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && has) {
            cudaMemPoolProps props{};
            props.allocType = cudaMemAllocationTypePinned;
            props.handleTypes = cudaMemHandleTypeNone;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            DevPool *p = new DevPool;
            uint64_t all = UINT64_MAX;   // balance() returns what is too much
            if (cudaMemPoolCreate(&p->pool, &props) == cudaSuccess &&
                cudaMemPoolSetAttribute(p->pool, cudaMemPoolAttrReleaseThreshold, &all) == cudaSuccess &&
                cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking) == cudaSuccess) {
                if (cudaMalloc(&p->anchor, kWaitBuffer) != cudaSuccess) cudaGetLastError();
                pools[dev] = p;
            } else {
                cudaGetLastError();
                if (p->pool) cudaMemPoolDestroy(p->pool);
                delete p;
            }
        }
        tried[dev] = true;
    }
    out = pools[dev];
    return cudaSuccess;
}

// All work of the current device is done: cudaFree of a small buffer waits for it (5 us with the device idle, as long as
// cudaDeviceSynchronize takes). Unlike that call it may be made while a stream is captured in the relaxed mode,
// which a handle that goes must not end.
inline bool wait_for_device()
{
    void *p = nullptr;
    if (cudaMalloc(&p, kWaitBuffer) == cudaSuccess) return cudaFree(p) == cudaSuccess;
    cudaGetLastError();
    return cudaDeviceSynchronize() == cudaSuccess;
}

// what the current device's pool keeps unused goes back to the device
inline cudaError_t release_memory()
{
    DevPool *d = nullptr;
    if (cudaError_t e = device_pool(d)) return e;
    if (!d) return cudaSuccess;
    std::vector<std::pair<void *, size_t>> gone;
    {
        std::lock_guard<std::mutex> lock(d->mutex);
        gone.swap(d->kept);
        d->kept_bytes = 0;
    }
    cudaError_t err = cudaSuccess;
    auto note = [&err](cudaError_t e) {
        if (e && !err) err = e;
    };
    for (auto &b : gone) {
        const cudaError_t e = cudaFree(b.first);
        note(e);
        if (e) {   // a capture that forbids it: for the next time
            std::lock_guard<std::mutex> lock(d->mutex);
            d->kept.push_back(b);
            d->kept_bytes += b.second;
        }
    }
    note(cudaStreamSynchronize(d->stream));   // the releases on it are then done
    note(cudaMemPoolTrimTo(d->pool, 0));
    return err;
}

// bytes of device memory on the current device, for every stream
inline cudaError_t dev_alloc(void **p, size_t bytes)
{
    DevPool *d = nullptr;
    if (cudaError_t e = device_pool(d)) return e;
    if (!d) return cudaMalloc(p, bytes);
    const bool large = bytes > kPoolBuffer;
    if (large) {
        bytes = (bytes + (size_t(2) << 20) - 1) >> 21 << 21;
        std::lock_guard<std::mutex> lock(d->mutex);
        auto best = d->kept.end();   // the smallest that is large enough, at most a quarter more
        for (auto b = d->kept.begin(); b != d->kept.end(); ++b)
            if (b->second >= bytes && b->second <= bytes + bytes / 4 && (best == d->kept.end() || b->second < best->second))
                best = b;
        if (best != d->kept.end()) {
            *p = best->first;
            d->held.insert(*best);
            d->kept_bytes -= best->second;
            d->kept.erase(best);
            return cudaSuccess;
        }
    }
    auto take = [&] { return large ? cudaMalloc(p, bytes) : cudaMallocFromPoolAsync(p, bytes, d->pool, d->stream); };
    cudaError_t e = take();
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        release_memory();
        e = take();
    }
    if (e) return e;
    if (!large) return cudaStreamSynchronize(d->stream);
    try {
        std::lock_guard<std::mutex> lock(d->mutex);
        d->held.emplace(*p, bytes);
    } catch (const std::bad_alloc &) {
        cudaFree(*p);
        throw;
    }
    return cudaSuccess;
}

// While one lives, its thread's releases on the device that was current when it was made wait for the device once, at the first
// of them: for a handle that goes, with nothing enqueued in between (720p, window 64: 185 us with a wait for
// each of its buffers, 139 so).
class DevRelease {
public:
    DevRelease() : outer_(current())
    {
        device_pool(pool_);
        current() = this;
    }
    ~DevRelease()
    {
        current() = outer_;
        try {
            if (any_) pool_->balance(large_);
        } catch (const std::bad_alloc &) {   // no room for its list: another release does it
        }
    }
    DevRelease(const DevRelease &) = delete;
    DevRelease &operator=(const DevRelease &) = delete;

    // a release to pool d: whether all work before it is done
    static bool wait(DevPool *d)
    {
        DevRelease *r = current();
        if (!r || r->pool_ != d) return wait_for_device();
        return r->waited_ = r->waited_ || wait_for_device();
    }
    // a small buffer went to pool d's stream, or a large one is kept
    static void released(DevPool *d, bool large)
    {
        DevRelease *r = current();
        if (r && r->pool_ == d) {
            r->any_ = true;
            r->large_ = r->large_ || large;
        } else {
            d->balance(large);
        }
    }

private:
    static DevRelease *&current()
    {
        static thread_local DevRelease *r = nullptr;
        return r;
    }
    DevRelease *outer_;
    DevPool *pool_ = nullptr;
    bool waited_ = false, any_ = false, large_ = false;
};

// after all work of the memory's device
inline void dev_free(void *p) noexcept
try {
    if (!p) return;
    cudaPointerAttributes at{};
    int cur = 0;
    if (cudaGetDevice(&cur) != cudaSuccess || cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();   // the runtime is shutting down: the process's memory goes with it
        return;
    }
    const bool other = at.device != cur;
    if (other) cudaSetDevice(at.device);
    DevPool *d = nullptr;
    const cudaError_t e = device_pool(d);
    if (!e && !d) {
        cudaFree(p);
    } else if (e || !DevRelease::wait(d)) {
        cudaGetLastError();   // a capture that forbids it or a failed context: the memory stays, since work may still read it
    } else {
        std::vector<std::pair<void *, size_t>> gone;   // given back outside the lock
        bool large = false, kept = false;
        {
            std::lock_guard<std::mutex> lock(d->mutex);
            const auto b = d->held.find(p);
            large = b != d->held.end();
            if (large) {
                const std::pair<void *, size_t> buffer = *b;
                kept = buffer.second <= kLargeKeep;
                if (kept) {
                    d->drop(kLargeKeep - buffer.second, gone);
                    d->kept.push_back(buffer);
                    d->kept_bytes += buffer.second;
                } else {
                    gone.push_back(buffer);
                }
                d->held.erase(b);
            }
        }
        for (auto &b : gone) cudaFree(b.first);
        if (!large) cudaFreeAsync(p, d->stream);
        if (!large || kept) DevRelease::released(d, kept);
    }
    if (other) cudaSetDevice(cur);
} catch (const std::bad_alloc &) {   // no room for the lists: the memory stays
}

}   // namespace b200
