// ap_batch_map.cuh -- the order in which the batch queue runs through a tile (host and device).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define AP_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define AP_HOST_DEVICE inline
#endif

namespace ap {

// Pixel q (0..255) of item `item` of a tile of `patches` patches of 256 pixels -> its patch, and its place
// w (0..255) there.  The groups of 32 pixels are taken in a scattered order (a multiplier coprime to their
// number).  64 bits: a tile of one column of 2^31 - 1 pixels in patches of 256 x 1 has 2^31 - 1 patches,
// 2^34 groups.
AP_HOST_DEVICE int64_t batch_scatter(int64_t patches, int64_t item, int q, int* w) {
    const uint64_t groups = (uint64_t)patches * 8;
    uint64_t g = (uint64_t)item * 8 + (uint64_t)(q >> 5);
    if (patches % 7919) g = g * 7919 % groups;  // 7919 is an odd prime
    *w = (int)(g & 7) * 32 + (q & 31);
    return (int64_t)(g >> 3);
}

}  // namespace ap
