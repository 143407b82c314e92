// The library's device allocations (csrc/memory.cpp) on the CPU, against a fake of
// the runtime: a device of 1 000 bytes and a working pool that keeps 400 of them
// unused until it is trimmed.  Allocations that fit only without the kept bytes
// must succeed, errors of other kinds and real shortage must come back as they
// are, and nothing may be waited for while a stream is captured.
#include <cstdio>
#include <cstdlib>

#include "tch_internal.cuh"

static size_t g_used = 0, g_kept = 0, g_trims = 0, g_syncs = 0, g_calls = 0;
static cudaError_t g_forced = cudaSuccess, g_last = cudaSuccess;
static bool g_capturing = false;
static int g_pool_tag;

static cudaError_t take(void** p, size_t bytes) {
    g_calls++;
    if (g_forced != cudaSuccess) return g_last = g_forced;
    if (g_used + g_kept + bytes > 1000) return g_last = cudaErrorMemoryAllocation;
    g_used += bytes;
    *p = &g_pool_tag;
    return cudaSuccess;
}

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes) { return take(p, bytes); }
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t) { return take(p, bytes); }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t bytes, cudaMemPool_t, cudaStream_t) { return take(p, bytes); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* pool, const cudaMemPoolProps*) {
    *pool = reinterpret_cast<cudaMemPool_t>(&g_pool_tag);
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr a, void* v) {
    *static_cast<unsigned long long*>(v) = a == cudaMemPoolAttrReservedMemCurrent ? g_kept + 10 : 10;
    return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) {
    g_trims++;
    g_kept = 0;
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    *f = 1000 - g_used - g_kept;
    *t = 1000;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    g_syncs++;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
}

#define REQUIRE(x)                                                    \
    do {                                                              \
        if (!(x)) {                                                   \
            printf("line %d: %s\n", __LINE__, #x);                    \
            return 1;                                                 \
        }                                                             \
    } while (0)

static void reset(size_t used, size_t kept) {
    g_used = used;
    g_kept = kept;
    g_trims = g_syncs = g_calls = 0;
    g_forced = g_last = cudaSuccess;
    g_capturing = false;
}

int main() {
    cudaMemPool_t pool = nullptr;
    REQUIRE(tch::working_pool(0, &pool) == cudaSuccess && pool);
    REQUIRE(tch::working_pool(-1, &pool) == cudaErrorInvalidDevice);
    REQUIRE(tch::working_pool(0, &pool) == cudaSuccess);
    for (int how = 0; how < 3; how++) {
        auto alloc = [&](size_t bytes) {
            int* p = nullptr;
            return how == 0 ? tch::device_alloc(&p, bytes) : tch::pool_alloc(&p, bytes, how == 1 ? pool : nullptr, nullptr);
        };
        reset(100, 400);  // fits as it is: nothing is given back
        REQUIRE(alloc(500) == cudaSuccess && g_trims == 0 && g_syncs == 0 && g_calls == 1);
        reset(100, 400);  // fits without the kept bytes
        REQUIRE(alloc(700) == cudaSuccess && g_trims == 1 && g_calls == 2 && g_used == 800);
        REQUIRE(g_last == cudaSuccess);  // no error of the first attempt is left behind
        reset(100, 400);  // does not fit at all
        REQUIRE(alloc(950) == cudaErrorMemoryAllocation && g_trims == 1 && g_calls == 2);
        reset(0, 400);  // another error
        g_forced = cudaErrorInvalidValue;
        REQUIRE(alloc(1) == cudaErrorInvalidValue && g_trims == 0 && g_calls == 1);
        reset(100, 400);  // under capture
        g_capturing = true;
        if (how > 0) REQUIRE(alloc(700) == cudaErrorMemoryAllocation && g_trims == 0 && g_syncs == 0);
    }
    reset(100, 400);  // the kept bytes count as free
    size_t f = 0;
    REQUIRE(tch::free_memory(0, &f) == cudaSuccess && f == 900);
    printf("memory ok\n");
    return 0;
}
