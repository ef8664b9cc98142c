// scratch.cpp - stream-ordered device scratch.
#include <cuda_runtime.h>
#include <string.h>

#include <mutex>

#include "internal.h"

namespace cumf {

// One pool per device that keeps up to 256 MB between calls (the default pool returns its memory
// at every synchronisation, and mapping it again cost more than the warm start's feature kernels
// at 50,000 users).  Allocations are ordered on their stream, so any number of threads and
// streams may use the pool at once.
cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s) {
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaMallocAsync(p, bytes, s);
    cudaMemPool_t pool;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!pools[dev]) {
            cudaMemPoolProps props;
            memset(&props, 0, sizeof(props));
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            cudaMemPool_t made;
            if ((e = cudaMemPoolCreate(&made, &props)) != cudaSuccess) return e;
            uint64_t keep = 256ull << 20;
            if ((e = cudaMemPoolSetAttribute(made, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
                cudaMemPoolDestroy(made);
                return e;
            }
            pools[dev] = made;
        }
        pool = pools[dev];
    }
    return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

}  // namespace cumf
