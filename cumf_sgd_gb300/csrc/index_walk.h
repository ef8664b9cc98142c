// index_walk.h - grid-stride walks over up to 2^32 entries.
//
// Shared by device code and host tests.
#pragma once
#include <stdint.h>

#ifndef CUMF_HD
#ifdef __CUDACC__
#define CUMF_HD __host__ __device__ __forceinline__
#else
#define CUMF_HD inline
#endif
#endif

namespace cumf {

// f(first), f(first + step), ... below count, `kUnroll` at a time.  The steps are counted: the index
// compared with count would wrap where it passes 2^32 - step and the walk never end.
template <int kUnroll = 1, class F>
CUMF_HD void index_walk(uint32_t first, uint32_t step, uint32_t count, F &&f) {
    uint32_t left = first < count ? (count - first - 1) / step + 1 : 0;
#pragma unroll kUnroll
    for (uint32_t i = first; left > 0; --left, i += step) f(i);
}

}  // namespace cumf
