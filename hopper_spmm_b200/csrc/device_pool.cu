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

// What an upload uses; the next one finds it there.
struct Staging {
    char *pinned = nullptr;  // [kUploadThreads][2][kUploadChunk]
    int device = -1;         // of the streams and events
    cudaStream_t stream[kUploadThreads] = {};
    cudaEvent_t done[kUploadThreads][2] = {};
    void release_streams() {
        for (int t = 0; t < kUploadThreads; ++t) {
            for (cudaEvent_t &d : done[t]) {
                if (d) cudaEventDestroy(d);
                d = nullptr;
            }
            if (stream[t]) cudaStreamDestroy(stream[t]);
            stream[t] = nullptr;
        }
        device = -1;
    }
    void release() {
        release_streams();
        if (pinned) cudaFreeHost(pinned);
        pinned = nullptr;
    }
    // For the current device.  Leaves nothing behind when it fails.
    cudaError_t open(int current) {
        cudaError_t e = cudaSuccess;
        if (!pinned) e = cudaHostAlloc(reinterpret_cast<void **>(&pinned), kUploadThreads * 2 * kUploadChunk, cudaHostAllocPortable);
        if (e != cudaSuccess) pinned = nullptr;
        if (e == cudaSuccess && device != current) {
            release_streams();
            for (int t = 0; t < kUploadThreads && e == cudaSuccess; ++t) {
                e = cudaStreamCreateWithFlags(&stream[t], cudaStreamNonBlocking);
                for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = cudaEventCreateWithFlags(&done[t][k], cudaEventDisableTiming);
            }
            device = current;
        }
        if (e != cudaSuccess) release();
        return e;
    }
};
std::mutex g_staging_lock;
Staging g_staging;

}  // namespace

cudaError_t upload_pageable(void *dst, const void *src, size_t bytes) {
    std::unique_lock<std::mutex> guard(g_staging_lock, std::defer_lock);
    if (bytes < 4 * kUploadChunk || !guard.try_lock()) return cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (g_staging.open(device) != cudaSuccess) {
        cudaGetLastError();
        return cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    }
    e = cudaStreamSynchronize(nullptr);  // whatever was queued before the copy is done before it
    if (e != cudaSuccess) return e;
    std::atomic<size_t> next{0};
    std::atomic<int> failed{(int)cudaSuccess};
    auto worker = [&](int t) {
        auto ok = [&](cudaError_t r) {
            if (r != cudaSuccess) failed = (int)r;
            return r == cudaSuccess;
        };
        if (!ok(cudaSetDevice(device))) return;
        for (int k = 0; failed == (int)cudaSuccess; k ^= 1) {
            const size_t at = next.fetch_add(kUploadChunk);
            if (at >= bytes) break;
            const size_t n = std::min(kUploadChunk, bytes - at);
            char *buf = g_staging.pinned + (size_t)(2 * t + k) * kUploadChunk;
            if (!ok(cudaEventSynchronize(g_staging.done[t][k]))) break;  // (at once for one not recorded since the last upload)
            std::memcpy(buf, static_cast<const char *>(src) + at, n);
            if (!ok(cudaMemcpyAsync(static_cast<char *>(dst) + at, buf, n, cudaMemcpyHostToDevice, g_staging.stream[t])) ||
                !ok(cudaEventRecord(g_staging.done[t][k], g_staging.stream[t])))
                break;
        }
        ok(cudaStreamSynchronize(g_staging.stream[t]));
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
        g_staging.release();
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
