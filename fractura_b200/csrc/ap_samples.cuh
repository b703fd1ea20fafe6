// ap_samples.cuh -- the order of the samples of a supersampling pass (host and device).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define AP_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define AP_HOST_DEVICE inline
#endif

namespace ap {

// The samples of pixels of f x f each, pixel after pixel and row after row, run in parts of whole rows whose
// samples 31 bits number (f is below 2^25): 32 pixels at f = 8192 have 2^31 of them.
AP_HOST_DEVICE int sample_rows(int f) {  // rows of a part
    return (1 << 30) / f;
}

// Sample q of the part that starts at row `row0` -> its pixel and its place (sx, sy) there.
AP_HOST_DEVICE void sample_place(int row0, int q, int f, int* pixel, int* sx, int* sy) {
    const int row = row0 + (int)((unsigned)q / (unsigned)f);
    *sx = (int)((unsigned)q % (unsigned)f);
    *pixel = (int)((unsigned)row / (unsigned)f);
    *sy = (int)((unsigned)row % (unsigned)f);
}

}  // namespace ap
