#include "device_pool.hpp"

#include <cstdint>
#include <mutex>

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

}  // namespace

cudaError_t pool_alloc_bytes(void **out, size_t bytes, cudaStream_t stream) {
    *out = nullptr;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    cudaMemPool_t pool = nullptr;
    if (e == cudaSuccess) e = pool_of(device, &pool);
    if (e != cudaSuccess) return e;
    e = cudaMallocFromPoolAsync(out, bytes, pool, stream);
    if (e == cudaErrorMemoryAllocation) {  // what was freed may still be waiting for its stream, or be kept
        cudaGetLastError();
        cudaDeviceSynchronize();
        cudaMemPoolTrimTo(pool, 0);
        e = cudaMallocFromPoolAsync(out, bytes, pool, stream);
    }
    return e;
}

void pool_free(void *ptr, cudaStream_t stream) {
    if (ptr) cudaFreeAsync(ptr, stream);
}

cudaError_t pool_release(int device) {
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
