// Device memory of formats, plans and their construction.
//
// cudaMalloc and cudaFree map and unmap memory and stop the device; a conversion makes two dozen buffers, and a
// caller with a new matrix per step (a sampled graph) paid ten milliseconds for them.  They come from one CUDA
// memory pool per device instead, which keeps at most kPoolKeepBytes of freed memory for the next object and
// gives the rest back to the driver at the next synchronisation; b200spmm_release_cached_memory gives back all
// of it, and so does an allocation that finds the device full.  The pool is the driver's: it may be used from
// any thread, and what one stream frees another one gets only when the order of their work allows it.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cuda_runtime.h>

namespace b200spmm {

// A buffer of kPoolMaxBytes or more is the driver's own (cudaMalloc, cudaFree): the pool would not keep it, and maps
// new memory several times more slowly (graph of 2^24 nodes, 35 GB in all: 930 ms of conversion against 100).
constexpr size_t kPoolMaxBytes = (size_t)128 << 20;

// Enough for the working set of a matrix of some ten million entries, 0.3 % of the card.
constexpr size_t kPoolKeepBytes = (size_t)512 << 20;

cudaError_t pool_alloc_bytes(void **out, size_t bytes, cudaStream_t stream);
// Memory that is there at once, while a stream is being captured too: the driver's own, whatever its size.
cudaError_t pool_alloc_under_capture(void **out, size_t bytes);
// What was queued on `stream` may still use the memory; a large buffer is given back when the device is idle.
void pool_free(void *ptr, cudaStream_t stream = nullptr);
cudaError_t pool_release(int device);

// Memory of the current device, usable by work that is ordered after `stream`.
template <typename T>
cudaError_t pool_alloc(T **out, size_t count, cudaStream_t stream = nullptr) {
    void *p = nullptr;
    const cudaError_t e = pool_alloc_bytes(&p, std::max<size_t>(count * sizeof(T), 16), stream);
    *out = static_cast<T *>(p);
    return e;
}

// Copies `bytes` from pageable host memory to the current device and waits for it.  The driver's own copy moves 11
// GB/s, one thread filling its staging buffer; here kUploadThreads threads fill pinned buffers of their own (16 MB
// in all) over streams of their own, which keeps the link at 40-50 GB/s.  Buffers, streams and events are kept for the next
// upload until b200spmm_release_cached_memory, the latter for one device at a time: made anew they were 0.8 of the 5.0 ms that the
// plan of a matrix of 108 MB took.  8 or 12 threads are no faster.
// Small copies, and uploads while another one holds the buffers, go the driver's way.
constexpr int kUploadThreads = 4;
constexpr size_t kUploadChunk = (size_t)2 << 20;
cudaError_t upload_pageable(void *dst, const void *src, size_t bytes);

// Buffers that are needed while an object is built, released on every exit path.  Small ones share blocks of
// kBlockBytes: two dozen calls of the driver, each way, were a tenth of a small conversion.
struct PoolScratch {
    static constexpr size_t kBlockBytes = (size_t)8 << 20;
    cudaStream_t stream = nullptr;
    void *ptrs[24] = {};
    int n = 0;
    char *block = nullptr;  // the current block's free part
    size_t left = 0;
    explicit PoolScratch(cudaStream_t s = nullptr) : stream(s) {}
    PoolScratch(const PoolScratch &) = delete;
    template <typename T>
    cudaError_t alloc(T **out, size_t count) {
        const size_t bytes = (std::max<size_t>(count * sizeof(T), 16) + 255) & ~(size_t)255;
        *out = nullptr;
        const bool shared = bytes <= kBlockBytes / 2;
        if (!shared || left < bytes) {
            if (n == 24) return cudaErrorMemoryAllocation;
            void *p = nullptr;
            const cudaError_t e = pool_alloc_bytes(&p, shared ? kBlockBytes : bytes, stream);
            if (e != cudaSuccess) return e;
            ptrs[n++] = p;
            if (!shared) {
                *out = static_cast<T *>(p);
                return e;
            }
            block = static_cast<char *>(p);
            left = kBlockBytes;
        }
        *out = reinterpret_cast<T *>(block);
        block += bytes;
        left -= bytes;
        return cudaSuccess;
    }
    ~PoolScratch() { for (int i = 0; i < n; ++i) pool_free(ptrs[i], stream); }
};

}  // namespace b200spmm
