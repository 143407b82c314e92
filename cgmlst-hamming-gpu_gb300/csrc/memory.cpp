// Device memory of the library: the kept working pool, and allocations that take
// back what it keeps unused before they fail.

#include <mutex>

#include "tch_internal.cuh"

namespace tch {

// Working memory for building solvers, from a stream-ordered pool per device that
// keeps up to 512 MB between calls (mapping it anew took a millisecond of a small
// set's encoding); the driver hands back what is above that when the stream that
// freed it is next waited for.
cudaError_t working_pool(int device, cudaMemPool_t* out) {
    constexpr uint64_t kKeptBytes = (uint64_t)512 << 20;
    static std::mutex mu;
    static cudaMemPool_t pools[kMaxDevices] = {};
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(mu);
    if (!pools[device]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool;
        cudaError_t e = cudaMemPoolCreate(&pool, &props);
        if (e != cudaSuccess) return e;
        uint64_t keep = kKeptBytes;
        e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) return e;
        pools[device] = pool;
    }
    *out = pools[device];
    return cudaSuccess;
}

// The current device's working pool keeps nothing any more that is not in use.
static bool give_back() {
    int device = 0;
    cudaMemPool_t pool;
    return cudaGetDevice(&device) == cudaSuccess && working_pool(device, &pool) == cudaSuccess &&
           cudaDeviceSynchronize() == cudaSuccess && cudaMemPoolTrimTo(pool, 0) == cudaSuccess;
}

cudaError_t device_alloc(void** p, size_t bytes) {
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation || !give_back()) return e;
    cudaGetLastError();  // of the attempt that failed
    return cudaMalloc(p, bytes);
}

cudaError_t pool_alloc(void** p, size_t bytes, cudaMemPool_t pool, cudaStream_t st) {
    auto attempt = [&] {
        return pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaMallocAsync(p, bytes, st);
    };
    const cudaError_t e = attempt();
    if (e != cudaErrorMemoryAllocation) return e;
    cudaStreamCaptureStatus cs;  // nothing may be waited for while the stream is captured
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone || !give_back()) return e;
    cudaGetLastError();
    return attempt();
}

cudaError_t free_memory(int device, size_t* out) {
    size_t f = 0, t = 0;
    uint64_t reserved = 0, used = 0;
    cudaMemPool_t pool;
    const cudaError_t e = cudaMemGetInfo(&f, &t);
    if (e == cudaSuccess && working_pool(device, &pool) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) == cudaSuccess &&
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess && reserved > used)
        f += (size_t)(reserved - used);
    *out = f;
    return e;
}

}  // namespace tch
