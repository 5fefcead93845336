"""
The bookkeeping of the handles' device memory (slipcam_b200/csrc/dev_pool.h) against a stand-in for the CUDA runtime:
what is kept and for how long, running out of memory, captures that forbid a release, several threads.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'slipcam_b200', 'csrc')

RUNTIME = r'''
#pragma once
// A device of `capacity` bytes. Buffers are host addresses that are never used again. Releases on the pool's stream
// come about when it is synchronized; the pool then returns what is unused while it holds more than its threshold.
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorInvalidValue = 1, cudaErrorStreamCaptureUnsupported = 900 };
enum { cudaDevAttrMemoryPoolsSupported, cudaMemAllocationTypePinned, cudaMemHandleTypeNone, cudaMemLocationTypeDevice,
       cudaMemPoolAttrReleaseThreshold, cudaMemPoolAttrUsedMemCurrent, cudaMemPoolAttrReservedMemCurrent, cudaStreamNonBlocking };
struct Fake {
    std::mutex m;
    size_t capacity = size_t(4) << 30, direct = 0, pooled = 0, unused = 0, pending = 0, threshold = 0;
    uintptr_t next = 4096;
    std::map<void *, size_t> live_direct, live_pool;
    int mallocs = 0, waits = 0, pool_new = 0, device_syncs = 0;
    bool forbid = false, pools = true;
    size_t mapped() const { return direct + pooled; }
    void trim(size_t keep)
    {
        const size_t n = pooled > keep ? (unused < pooled - keep ? unused : pooled - keep) : 0;
        pooled -= n;
        unused -= n;
    }
};
inline Fake &fake() { static Fake f; return f; }
struct cudaMemPoolProps { int allocType, handleTypes; struct { int type, id; } location; };
struct cudaPointerAttributes { int device; };
typedef int *cudaMemPool_t;
typedef int *cudaStream_t;
inline cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaDeviceGetAttribute(int *v, int, int) { *v = fake().pools; return cudaSuccess; }
inline cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { *p = new int; return cudaSuccess; }
inline cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
inline cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, int, void *v) { fake().threshold = *static_cast<uint64_t *>(v); return cudaSuccess; }
inline cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, int what, void *v)
{
    Fake &f = fake();
    std::lock_guard<std::mutex> l(f.m);
    *static_cast<uint64_t *>(v) = what == cudaMemPoolAttrReservedMemCurrent ? f.pooled : f.pooled - f.unused;
    return cudaSuccess;
}
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, int) { *s = new int; return cudaSuccess; }
inline cudaError_t cudaMalloc(void **p, size_t n)
{
    Fake &f = fake();
    std::lock_guard<std::mutex> l(f.m);
    if (f.forbid) return cudaErrorStreamCaptureUnsupported;
    if (f.mapped() + n > f.capacity) return cudaErrorMemoryAllocation;
    f.direct += n;
    f.mallocs += n > 256;
    f.waits += n <= 256;
    *p = reinterpret_cast<void *>(f.next += 256);
    f.live_direct[*p] = n;
    return cudaSuccess;
}
template <class T> cudaError_t cudaMalloc(T **p, size_t n) { return cudaMalloc(reinterpret_cast<void **>(p), n); }
inline cudaError_t cudaFree(void *p)
{
    Fake &f = fake();
    std::lock_guard<std::mutex> l(f.m);
    if (f.forbid) return cudaErrorStreamCaptureUnsupported;
    auto b = f.live_direct.find(p);
    if (b == f.live_direct.end()) std::abort();   // not a buffer of cudaMalloc's, or freed twice
    f.direct -= b->second;
    f.live_direct.erase(b);
    return cudaSuccess;
}
inline cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t)
{
    Fake &f = fake();
    std::lock_guard<std::mutex> l(f.m);
    if (f.unused >= n) {
        f.unused -= n;
    } else {
        if (f.mapped() + n > f.capacity) return cudaErrorMemoryAllocation;
        f.pooled += n;
        ++f.pool_new;
    }
    *p = reinterpret_cast<void *>(f.next += 256);
    f.live_pool[*p] = n;
    return cudaSuccess;
}
inline cudaError_t cudaFreeAsync(void *p, cudaStream_t)
{
    Fake &f = fake();
    std::lock_guard<std::mutex> l(f.m);
    auto b = f.live_pool.find(p);
    if (b == f.live_pool.end()) std::abort();
    f.pending += b->second;
    f.live_pool.erase(b);
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    Fake &f = fake();
    std::lock_guard<std::mutex> l(f.m);
    f.unused += f.pending;
    f.pending = 0;
    f.trim(f.threshold);
    return cudaSuccess;
}
inline cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t keep)
{
    Fake &f = fake();
    std::lock_guard<std::mutex> l(f.m);
    f.trim(keep);
    return cudaSuccess;
}
inline cudaError_t cudaDeviceSynchronize() { ++fake().device_syncs; return fake().forbid ? cudaErrorStreamCaptureUnsupported : cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { a->device = 0; return cudaSuccess; }
'''

PROGRAM = r'''
#include "dev_pool.h"
#include <cstdio>
#include <cstring>
#include <set>
#include <thread>
using namespace b200;
constexpr size_t MB = size_t(1) << 20;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
static void *get(size_t n) { void *p = nullptr; return dev_alloc(&p, n) == cudaSuccess ? p : nullptr; }

int main(int, char **argv)
{
    Fake &f = fake();
    const auto test = [&](const char *name) { return std::strcmp(argv[1], name) == 0; };
    if (test("reuse")) {   // a handle's buffers are there for the next handle; others are not taken for them
        for (int i = 0; i < 3; ++i) {
            void *a = get(300 * MB), *b = get(300 * MB + 1000), *c = get(3 * MB), *d = get(1);
            CHECK(a && b && c && d && a != b);
            dev_free(d), dev_free(c), dev_free(b), dev_free(a);
        }
        CHECK(f.mallocs == 2 && f.pool_new == 2);
        void *a = get(100 * MB);
        CHECK(f.mallocs == 3);
        dev_free(a);
        release_memory();
        f.pool_new = 0;   // small handles side by side, again and again: their buffers stay, whatever is in use
        for (int i = 0; i < 4; ++i) {
            void *s[4][3];
            for (auto &h : s)
                for (void *&p : h) p = get(30 * MB);
            for (auto &h : s)
                for (void *p : h) dev_free(p);
        }
        CHECK(f.pool_new <= 12);
        void *big[3] = {get(290 * MB), get(290 * MB), get(290 * MB)};   // and after a large handle: its buffers make room
        for (void *p : big) dev_free(p);
        f.pool_new = 0;
        for (int i = 0; i < 4; ++i) {
            void *s[4][3];
            for (auto &h : s)
                for (void *&p : h) p = get(30 * MB);
            for (auto &h : s)
                for (void *p : h) dev_free(p);
            CHECK(f.mapped() <= 1024 * MB + 256);
        }
        CHECK(f.pool_new <= 12);
        void *a2 = get(290 * MB);
        CHECK(f.mallocs == 6 && a2);   // the last released is still there
        dev_free(a2);
    } else if (test("bound")) {   // at most 1 GiB stays, also of buffers that are each well below it, at once
        for (size_t n : {1 * MB, 30 * MB, 60 * MB, 250 * MB, 900 * MB}) {
            std::vector<void *> p;
            for (size_t k = 0; k < 2500 * MB / n; ++k) p.push_back(get(n));
            for (void *q : p) {
                CHECK(q);
                dev_free(q);
            }
            CHECK(f.mapped() <= 1024 * MB + 256);
        }
        CHECK(f.device_syncs == 0);
    } else if (test("full")) {   // out of memory: what is kept goes first, large buffers or small
        f.capacity = 1000 * MB;
        for (size_t n : {30 * MB, 200 * MB, 400 * MB})
            for (size_t want : {900 * MB, 20 * MB}) {
                std::vector<void *> p;
                for (size_t k = 0; k < 950 * MB / n; ++k) p.push_back(get(n));
                for (void *q : p) dev_free(q);
                p.clear();
                for (size_t k = 0; k < 980 * MB / want; ++k) {
                    p.push_back(get(want));
                    CHECK(p.back());
                }
                void *none = nullptr;
                CHECK(dev_alloc(&none, 900 * MB) == cudaErrorMemoryAllocation);
                for (void *q : p) dev_free(q);
            }
    } else if (test("release")) {
        void *p[4] = {get(400 * MB), get(100 * MB), get(10 * MB), get(1000 * MB)};
        for (void *q : p) dev_free(q);
        CHECK(f.mapped() >= 510 * MB);
        CHECK(release_memory() == cudaSuccess);
        CHECK(f.mapped() == 256);   // the anchor
        CHECK(get(400 * MB));
    } else if (test("forbidden")) {   // a capture forbids the wait: the memory is neither given back nor given out
        void *a = get(100 * MB), *b = get(MB), *k = get(200 * MB);
        dev_free(k);
        f.forbid = true;
        dev_free(a), dev_free(b);
        CHECK(release_memory() != cudaSuccess);
        f.forbid = false;
        CHECK(f.live_direct.count(a) && f.live_pool.count(b));
        void *c = get(100 * MB), *d = get(MB);
        CHECK(c != a && d != b);
        CHECK(release_memory() == cudaSuccess && !f.live_direct.count(k));
    } else if (test("together")) {   // a handle's buffers go after one wait, and the excess with them
        std::vector<void *> p;
        for (int k = 0; k < 20; ++k) p.push_back(get((10 + 90 * (k % 2)) * MB));
        f.waits = 0;
        {
            DevRelease all;
            for (void *q : p) dev_free(q);
            CHECK(f.waits == 1);
        }
        CHECK(f.mapped() <= 1024 * MB + 256);
        void *a = get(MB);
        dev_free(a);
        CHECK(f.waits == 2);
        void *b = get(100 * MB), *c = get(100 * MB);
        {
            DevRelease all;
            f.forbid = true;
            dev_free(b);   // forbidden: this one stays, the next waits anew
            f.forbid = false;
            dev_free(c);
        }
        CHECK(f.live_direct.count(b) && get(100 * MB) != b);
    } else if (test("none")) {   // a device without pools
        f.pools = false;
        void *a = get(100 * MB), *b = get(MB);
        dev_free(a), dev_free(b);
        CHECK(f.mapped() == 0 && release_memory() == cudaSuccess);
    } else if (test("threads")) {
        std::mutex m;
        std::set<void *> live;
        bool bad = false;
        auto work = [&](unsigned seed) {
            std::vector<void *> mine;
            for (int i = 0; i < 2000; ++i) {
                seed = seed * 1664525u + 1013904223u;
                if ((seed >> 16) % 2 || mine.empty()) {
                    void *p = get(((seed >> 20) % 80 + 1) * MB);
                    if (!p) continue;
                    std::lock_guard<std::mutex> l(m);
                    bad |= !live.insert(p).second;
                    mine.push_back(p);
                } else {
                    void *p = mine.back();
                    mine.pop_back();
                    {
                        std::lock_guard<std::mutex> l(m);
                        live.erase(p);
                    }
                    dev_free(p);
                }
            }
            for (void *p : mine) {
                {
                    std::lock_guard<std::mutex> l(m);
                    live.erase(p);
                }
                dev_free(p);
            }
        };
        std::vector<std::thread> t;
        for (unsigned i = 0; i < 6; ++i) t.emplace_back(work, i);
        for (auto &x : t) x.join();
        CHECK(!bad && f.mapped() <= 1024 * MB + 256);
        CHECK(release_memory() == cudaSuccess && f.mapped() == 256);
    } else {
        return 2;
    }
    return 0;
}
'''


@pytest.fixture(scope='module')
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp('dev_memory')
    (d / 'cuda_runtime.h').write_text(RUNTIME)
    (d / 'main.cpp').write_text(PROGRAM)
    subprocess.run(['g++', '-std=c++17', '-O1', '-g', '-pthread', '-I', str(d), '-I', CSRC, str(d / 'main.cpp'), '-o',
                    str(d / 'main')], check=True)
    return str(d / 'main')


@pytest.mark.parametrize('name', ['reuse', 'bound', 'full', 'release', 'forbidden', 'together', 'none', 'threads'])
def test_bookkeeping(program, name):
    r = subprocess.run([program, name], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
