// Device memory of the library's objects.
#pragma once
#include <cuda_runtime_api.h>

#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <set>

namespace rmdhost {

// gives back what the contexts of `device` keep; whether there was anything
inline bool giveBackKept(int device);

// What `attempt` returns: a call that may allocate on the current device, made
// again if the device is full while contexts keep free blocks of it.
template <class Attempt>
cudaError_t withKeptMemory(Attempt attempt) {
    cudaError_t e = attempt();
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();  // not for the next launch's check
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || !giveBackKept(device)) return e;
    if ((e = attempt()) == cudaErrorMemoryAllocation) cudaGetLastError();
    return e;
}
inline cudaError_t deviceAlloc(void **p, size_t n) {
    return withKeptMemory([&] { return cudaMalloc(p, n); });
}
inline cudaError_t loadLibrary(cudaLibrary_t *library, const void *code) {
    return withKeptMemory([&] { return cudaLibraryLoadData(library, code, nullptr, nullptr, 0, nullptr, nullptr, 0); });
}

// A context's device memory: blocks that its scenes, renderers and batches free
// stay with it for the next ones, up to kMemoryKept bytes; beyond that, and
// with the context and its last object, they go back to the device.  cudaMalloc
// and cudaFree of the 10-500 MB blocks that a scene and its renderer take cost
// 1-10 ms each, and now and then hundreds (the 852 k-triangle scene: 20 ms to
// 4 s of a creation).  A driver pool maps its memory anew whenever a block fits
// no hole (2-3 ms for the tree's workspace and for the paths, in one of four
// creations 40-1,200 ms); a kept block is handed out as it is.  Sizes below
// 1 GiB are rounded up to an eighth of their power of two, so that a scene a
// little larger than the one before takes the same blocks; a size that only fits
// as it is gets such a block, which is not kept.  Any thread may
// allocate and free.  Kept blocks are free memory to every allocation of the
// library: one that finds the device full has all contexts of the device give
// theirs back (withKeptMemory).
//
// A context's blocks are used on its stream alone, so what is enqueued on a block
// comes after all that its last owner enqueued, waited for or not (cudaFree waits
// by itself).  No wait stands in an object's end: it would have to be for a stream
// or a device that another thread may be capturing on, which refuses it and spoils
// the capture.
struct DevPool {
    static constexpr size_t kMemoryKept = size_t(2) << 30;
    const int device;
    std::mutex mutex;
    std::multimap<size_t, void *> kept;  // free blocks by size
    size_t keptBytes = 0;
    std::set<void *> unrounded;  // blocks in use that are smaller than their rounded size
    explicit DevPool(int device);
    ~DevPool();
    DevPool(const DevPool &) = delete;
    DevPool &operator=(const DevPool &) = delete;
    static size_t rounded(size_t n) {
        size_t step = 512;
        if (n < (size_t(1) << 30))
            while (step * 16 <= n) step *= 2;
        return (n + step - 1) / step * step;
    }
    // a block of the current device, which has to be the context's
    cudaError_t alloc(void **p, size_t n) {
        const size_t size = rounded(n);
        {
            std::lock_guard<std::mutex> lock(mutex);
            const auto it = kept.find(size);
            if (it != kept.end()) {
                *p = it->second;
                keptBytes -= size;
                kept.erase(it);
                return cudaSuccess;
            }
        }
        cudaError_t e = deviceAlloc(p, size);
        if (e == cudaErrorMemoryAllocation && n < size && (e = deviceAlloc(p, n)) == cudaSuccess) {
            std::lock_guard<std::mutex> lock(mutex);
            try {
                unrounded.insert(*p);
            } catch (const std::bad_alloc &) {
                cudaFree(*p);
                *p = nullptr;
                return cudaErrorMemoryAllocation;
            }
        }
        return e;
    }
    // takes back a block that alloc gave for n bytes
    void free(void *p, size_t n) noexcept {
        const size_t size = rounded(n);
        std::lock_guard<std::mutex> lock(mutex);
        if (unrounded.erase(p)) {
            cudaFree(p);
            return;
        }
        try {
            kept.emplace(size, p);
        } catch (const std::bad_alloc &) {  // objects free their buffers where nothing may be thrown
            cudaFree(p);
            return;
        }
        keptBytes += size;
        while (keptBytes > kMemoryKept) {  // the largest go first: small ones are asked for on every read-out
            const auto largest = std::prev(kept.end());
            cudaFree(largest->second);
            keptBytes -= largest->first;
            kept.erase(largest);
        }
    }
    // whether there were any
    bool giveBack() {
        std::lock_guard<std::mutex> lock(mutex);
        const bool any = !kept.empty();
        for (auto &block : kept) cudaFree(block.second);
        kept.clear();
        keptBytes = 0;
        return any;
    }
};

struct PoolList {
    std::mutex mutex;
    std::set<DevPool *> pools;
};
inline PoolList &poolList() {
    static PoolList *list = new PoolList;  // never destroyed: contexts may outlive this library's statics
    return *list;
}
inline DevPool::DevPool(int d) : device(d) {
    std::lock_guard<std::mutex> lock(poolList().mutex);
    poolList().pools.insert(this);
}
inline DevPool::~DevPool() {
    {
        std::lock_guard<std::mutex> lock(poolList().mutex);
        poolList().pools.erase(this);
    }
    giveBack();
}
inline bool giveBackKept(int device) {
    std::lock_guard<std::mutex> lock(poolList().mutex);
    bool any = false;
    for (DevPool *p : poolList().pools)
        if (p->device == device && p->giveBack()) any = true;
    return any;
}
// Free memory of the current device, the kept blocks included.
inline cudaError_t freeMemory(size_t &bytes) {
    size_t total = 0;
    int device = 0;
    cudaError_t e = cudaMemGetInfo(&bytes, &total);
    if (e != cudaSuccess || (e = cudaGetDevice(&device)) != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(poolList().mutex);
    for (DevPool *p : poolList().pools) {
        std::lock_guard<std::mutex> poolLock(p->mutex);
        if (p->device == device) bytes += p->keptBytes;
    }
    return e;
}

// Device buffer owned by a scene, renderer or batch, from its context's pool
// where one is set.  A new one may hold what a block's last owner left, so it is
// cleared and filled on the context's stream (the legacy stream is not ordered
// with it).
struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    std::shared_ptr<DevPool> from;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (ptr) {
            if (from) from->free(ptr, bytes);
            else cudaFree(ptr);
        }
        ptr = nullptr;
        bytes = 0;
    }
    cudaError_t alloc(size_t n) {
        release();
        bytes = n;
        if (n == 0) return cudaSuccess;
        return from ? from->alloc(&ptr, n) : deviceAlloc(&ptr, n);
    }
    void adopt(void *p, size_t n) {  // takes ownership of a block allocated as alloc(n) does
        release();
        ptr = p;
        bytes = n;
    }
    cudaError_t upload(const void *src, size_t n, cudaStream_t s) {
        cudaError_t e = alloc(n);
        if (e != cudaSuccess || n == 0) return e;
        e = cudaMemcpyAsync(ptr, src, n, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
        return cudaStreamSynchronize(s);
    }
    template <class T>
    T *as() const {
        return static_cast<T *>(ptr);
    }
};

}  // namespace rmdhost
