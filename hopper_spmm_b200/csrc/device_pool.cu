#include "device_pool.hpp"

#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <unordered_set>
#include <vector>

#include "../../include/b200_spmm.h"
#include "common.hpp"

namespace b200spmm {
namespace {

constexpr int kMaxDevices = 64;
std::mutex g_lock;
cudaMemPool_t g_pool[kMaxDevices] = {};

cudaError_t pool_of(int device, cudaMemPool_t *out) {
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> guard(g_lock);
    if (!g_pool[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        cudaError_t e = cudaMemPoolCreate(&pool, &props);
        if (e != cudaSuccess) return e;
        uint64_t keep = kPoolKeepBytes;
        e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return e;
        }
        g_pool[device] = pool;
    }
    *out = g_pool[device];
    return cudaSuccess;
}

std::mutex g_large_lock;
std::unordered_set<void *> g_large;  // the driver's own buffers: of kPoolMaxBytes and more, or allocated under a capture

std::mutex g_staging_lock;
void *g_staging = nullptr;  // [kUploadThreads][2][kUploadChunk] pinned bytes

}  // namespace

cudaError_t upload_pageable(void *dst, const void *src, size_t bytes) {
    std::unique_lock<std::mutex> guard(g_staging_lock, std::defer_lock);
    if (bytes < 4 * kUploadChunk || !guard.try_lock()) return cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    if (!g_staging && cudaHostAlloc(&g_staging, kUploadThreads * 2 * kUploadChunk, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        g_staging = nullptr;
        return cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    }
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);  // whatever was queued before the copy is done before it
    if (e != cudaSuccess) return e;
    std::atomic<size_t> next{0};
    std::atomic<int> failed{(int)cudaSuccess};
    auto worker = [&](int t) {
        cudaStream_t stream = nullptr;
        cudaEvent_t done[2] = {nullptr, nullptr};
        auto ok = [&](cudaError_t r) {
            if (r != cudaSuccess) failed = (int)r;
            return r == cudaSuccess;
        };
        if (ok(cudaSetDevice(device)) && ok(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking)) &&
            ok(cudaEventCreateWithFlags(&done[0], cudaEventDisableTiming)) && ok(cudaEventCreateWithFlags(&done[1], cudaEventDisableTiming))) {
            for (int k = 0; failed == (int)cudaSuccess; k ^= 1) {
                const size_t at = next.fetch_add(kUploadChunk);
                if (at >= bytes) break;
                const size_t n = std::min(kUploadChunk, bytes - at);
                char *buf = static_cast<char *>(g_staging) + (size_t)(2 * t + k) * kUploadChunk;
                if (!ok(cudaEventSynchronize(done[k]))) break;  // (at once for an event never recorded)
                std::memcpy(buf, static_cast<const char *>(src) + at, n);
                if (!ok(cudaMemcpyAsync(static_cast<char *>(dst) + at, buf, n, cudaMemcpyHostToDevice, stream)) ||
                    !ok(cudaEventRecord(done[k], stream)))
                    break;
            }
            ok(cudaStreamSynchronize(stream));
        }
        for (cudaEvent_t d : done)
            if (d) cudaEventDestroy(d);
        if (stream) cudaStreamDestroy(stream);
    };
    std::vector<std::thread> pool;
    pool.reserve(kUploadThreads);
    try {
        for (int t = 1; t < kUploadThreads; ++t) pool.emplace_back(worker, t);
    } catch (const std::system_error &) {  // no more threads to be had: those there are move all of it
    }
    worker(0);
    for (auto &th : pool) th.join();
    return (cudaError_t)failed.load();
}

cudaError_t pool_alloc_bytes(void **out, size_t bytes, cudaStream_t stream) {
    *out = nullptr;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    cudaMemPool_t pool = nullptr;
    if (e == cudaSuccess) e = pool_of(device, &pool);
    if (e != cudaSuccess) return e;
    auto allocate = [&]() { return bytes >= kPoolMaxBytes ? cudaMalloc(out, bytes) : cudaMallocFromPoolAsync(out, bytes, pool, stream); };
    e = allocate();
    if (e == cudaErrorMemoryAllocation) {  // what was freed may still be waiting for its stream, or be kept
        cudaGetLastError();
        cudaDeviceSynchronize();
        cudaMemPoolTrimTo(pool, 0);
        e = allocate();
    }
    if (e == cudaSuccess && bytes >= kPoolMaxBytes) {
        std::lock_guard<std::mutex> guard(g_large_lock);
        g_large.insert(*out);
    }
    return e;
}

cudaError_t pool_alloc_under_capture(void **out, size_t bytes) {
    *out = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // cudaMalloc is refused in the other modes; it is no part of the graph
    cudaError_t e = cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) return e;
    e = cudaMalloc(out, bytes);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> guard(g_large_lock);
        g_large.insert(*out);
    }
    return e;
}

void pool_free(void *ptr, cudaStream_t stream) {
    if (!ptr) return;
    bool large;
    {
        std::lock_guard<std::mutex> guard(g_large_lock);
        large = g_large.erase(ptr) != 0;
    }
    if (large) cudaFree(ptr);  // (waits for the device)
    else cudaFreeAsync(ptr, stream);
}

cudaError_t pool_release(int device) {
    {
        std::lock_guard<std::mutex> guard(g_staging_lock);
        if (g_staging) cudaFreeHost(g_staging);
        g_staging = nullptr;
    }
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> guard(g_lock);
        if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
        pool = g_pool[device];
    }
    return pool ? cudaMemPoolTrimTo(pool, 0) : cudaSuccess;
}

}  // namespace b200spmm

extern "C" int b200spmm_release_cached_memory(int device) {
    B200_CUDA_TRY(b200spmm::pool_release(device));
    return B200SPMM_OK;
}
