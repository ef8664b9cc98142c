// scratch.cpp - stream-ordered device scratch.
#include <cuda_runtime.h>
#include <string.h>

#include <mutex>

#include "internal.h"

namespace cumf {

namespace {

constexpr int kMaxDevices = 64;
constexpr uint64_t kKeepBytes = 256ull << 20;
std::mutex g_pool_mutex;
cudaMemPool_t g_pools[kMaxDevices] = {};

}  // namespace

// One pool per device that keeps up to 256 MB between calls: cudaMalloc and cudaFree took 0.17 of
// the 0.30 ms of an RMSE call on 1.4M ratings and 0.9 of the 1.4 ms of a ranking call, and the
// default pool returns its memory at every synchronisation.  Allocations are ordered on their
// stream, so any number of threads and streams may use the pool at once.
cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaMallocAsync(p, bytes, s);
    cudaMemPool_t pool;
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        if (!g_pools[dev]) {
            cudaMemPoolProps props;
            memset(&props, 0, sizeof(props));
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            cudaMemPool_t made;
            if ((e = cudaMemPoolCreate(&made, &props)) != cudaSuccess) return e;
            uint64_t keep = kKeepBytes;
            if ((e = cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
                cudaMemPoolDestroy(made);
                return e;
            }
            g_pools[dev] = made;
        }
        pool = g_pools[dev];
    }
    return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

void scratch_release() {
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    for (cudaMemPool_t pool : g_pools)
        if (pool && cudaMemPoolTrimTo(pool, 0) != cudaSuccess) cudaGetLastError();
}

}  // namespace cumf
