// dev_pool.h -- the device memory of the handles, from a CUDA memory pool of the library's own per device.
//
// A handle's buffers (for a 720p grid 14, some 900 MB with its tables) are mapped when it is made and unmapped
// when it goes, at 0.1 to 0.6 ms a buffer: more than the work of the calls that make a handle for one pass
// (the periodicity of one 720p frame: 4.5 of 7.5 ms). The pool keeps up to kPoolKeep bytes mapped for the
// next handle and returns what is above that to the device at its next synchronization; when the device is out
// of memory an allocation first returns all that is unused. The CUDA pool serves several threads and devices.
//
// The buffers are ready for, and freed after, every stream, as with cudaMalloc and cudaFree: an allocation
// waits for its (empty) stream, a release first for the device (wait_for_device). The contents of a buffer are
// undefined.
#pragma once

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <unordered_set>

#include <cuda_runtime.h>

namespace b200 {

constexpr uint64_t kPoolKeep = uint64_t(1) << 30;
// Larger buffers come from cudaMalloc: the pool could not keep two of them, and maps them more slowly (the 3.6 GB
// of spectra of a dense 1080p grid: a handle made in 27 ms from the pool, in 7 ms from cudaMalloc).
constexpr size_t kPoolBuffer = size_t(512) << 20;

constexpr size_t kWaitBuffer = 256;

struct DevPool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;   // orders the pool's allocations and releases; no work runs on it
    void *anchor = nullptr;          // keeps a block of small buffers mapped for wait_for_device
};

// the buffers above kPoolBuffer, so that a release knows them
struct DirectBuffers {
    std::mutex mutex;
    std::unordered_set<void *> held;
};
inline DirectBuffers &direct_buffers()
{
    static DirectBuffers *d = new DirectBuffers;   // outlives every handle
    return *d;
}

// the current device's pool (pool == nullptr: it has none), and the device's index
inline cudaError_t device_pool(DevPool &out, int &dev)
{
    static std::mutex mutex;
    static DevPool pools[64];
    static bool tried[64] = {};
    if (cudaError_t e = cudaGetDevice(&dev)) return e;
    out = DevPool{};
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
            uint64_t keep = kPoolKeep;
            DevPool p;
            if (cudaMemPoolCreate(&p.pool, &props) == cudaSuccess &&
                cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess &&
                cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) == cudaSuccess) {
                if (cudaMalloc(&p.anchor, kWaitBuffer) != cudaSuccess) cudaGetLastError();
                pools[dev] = p;
            } else {
                cudaGetLastError();
                if (p.pool) cudaMemPoolDestroy(p.pool);
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

// bytes of device memory on the current device, for every stream
inline cudaError_t dev_alloc(void **p, size_t bytes)
{
    DevPool d;
    int dev = 0;
    if (cudaError_t e = device_pool(d, dev)) return e;
    if (!d.pool) return cudaMalloc(p, bytes);
    if (bytes > kPoolBuffer) {
        cudaError_t e = cudaMalloc(p, bytes);
        if (e == cudaErrorMemoryAllocation) {   // what the pool holds unused first
            cudaGetLastError();
            cudaMemPoolTrimTo(d.pool, 0);
            e = cudaMalloc(p, bytes);
        }
        if (e) return e;
        DirectBuffers &b = direct_buffers();
        std::lock_guard<std::mutex> lock(b.mutex);
        b.held.insert(*p);
        return cudaSuccess;
    }
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, d.pool, d.stream);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        cudaStreamSynchronize(d.stream);
        cudaMemPoolTrimTo(d.pool, 0);
        e = cudaMallocFromPoolAsync(p, bytes, d.pool, d.stream);
    }
    return e ? e : cudaStreamSynchronize(d.stream);
}

// after all work of the memory's device
inline void dev_free(void *p)
{
    if (!p) return;
    cudaPointerAttributes at{};
    int cur = 0;
    if (cudaGetDevice(&cur) != cudaSuccess || cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();   // the runtime is shutting down: the process's memory goes with it
        return;
    }
    const bool other = at.device != cur;
    if (other) cudaSetDevice(at.device);
    DevPool d;
    int dev = 0;
    if (device_pool(d, dev) == cudaSuccess) {
        bool direct = !d.pool;
        if (!direct) {
            DirectBuffers &b = direct_buffers();
            std::lock_guard<std::mutex> lock(b.mutex);
            direct = b.held.erase(p) > 0;
        }
        if (direct)
            cudaFree(p);
        else if (wait_for_device())
            cudaFreeAsync(p, d.stream);
        else   // a capture that forbids it or a failed context: the memory stays, since work may still read it
            cudaGetLastError();
    }
    if (other) cudaSetDevice(cur);
}

}   // namespace b200
