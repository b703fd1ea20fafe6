// ap_samples.cuh -- the order of the samples of a supersampling pass (host and device).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define AP_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define AP_HOST_DEVICE inline
#endif

namespace ap {

// Sample q of pixels of f x f samples each, pixel after pixel, row after row -> its pixel and its place
// (sx, sy) there.  64 bits where the number of a sample needs them: 32 pixels at f = 8192 have 2^31.
AP_HOST_DEVICE void sample_place(int64_t q, int f, int* pixel, int* sx, int* sy) {
    if (q < INT32_MAX && f <= 46340) {  // f^2 < 2^31
        const unsigned f2 = (unsigned)f * (unsigned)f, sub = (unsigned)q % f2;
        *pixel = (int)((unsigned)q / f2);
        *sx = (int)(sub % (unsigned)f);
        *sy = (int)(sub / (unsigned)f);
    } else {
        const int64_t f2 = (int64_t)f * f, sub = q % f2;
        *pixel = (int)(q / f2);
        *sx = (int)(sub % f);
        *sy = (int)(sub / f);
    }
}

}  // namespace ap
