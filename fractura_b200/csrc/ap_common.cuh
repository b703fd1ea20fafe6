// ap_common.cuh -- shared device helpers of the B200 escape-time engine.
//
// Compiled with -fmad=false: no multiply-add is fused unless it is written
// with fma() below, so the arithmetic in the source is the arithmetic that
// runs (the escape step of a boundary pixel depends on it).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "apeiron_b200.h"

namespace ap {

// config.py:25-26
constexpr double kInvLn2 = 1.4426950408889634;
constexpr double kLnBailoutLog = 1.7129177284488854;
constexpr double kBailout = 65536.0;

// Error reporting of the C ABI (thread-local message).
void set_error(const char* fmt, ...);
int check_launch(const char* what);

// Coarse-pass perturbation kernel on packed inputs (ap_perturb_fast.cu);
// AP_E_UNSUPPORTED when the pass is not one it serves.
int launch_perturb_fast(const ApFrameParams& p, const ApFrameBuffers& b, cudaStream_t st);
int launch_perturb_fast_rows(const ApFrameParams& p, const ApFrameBuffers& b, int row0, int rows,
                             cudaStream_t st);

// FP32-mantissa FloatExp tier (ap_fe32.cu).
int launch_fe32(const ApFrameParams& p, const ApFrameBuffers& b, cudaStream_t st);

struct SampleOut {
    float s;      // float32 smooth value (reference storage type), -1 interior
    double s64;   // float64 smooth value
    int k;        // escape step, -1 = never escaped, -2 = cardioid/bulb skip
    int glitch;
    int iters;    // iterations stepped one at a time (work accounting)
    int leaps;    // BLA leaps taken
    int iters2;   // perturbation stage-2 direct steps
};

__device__ __forceinline__ SampleOut interior_sample() {
    SampleOut o;
    o.s = -1.0f;
    o.s64 = -1.0;
    o.k = -1;
    o.glitch = 0;
    o.iters = 0;
    o.leaps = 0;
    o.iters2 = 0;
    return o;
}

// Never escaped within max_iter iterations.
__device__ __forceinline__ SampleOut interior_after(int max_iter) {
    SampleOut o = interior_sample();
    o.iters = max_iter;
    return o;
}

// Pixel removed by the Mandelbrot cardioid/bulb test: interior, zero iterations.
__device__ __forceinline__ SampleOut skipped_sample() {
    SampleOut o = interior_sample();
    o.k = -2;
    return o;
}

// f32(k+1) - f32(nu), nu = (ln(ln|z|^2 / 2) - ln(8 ln 2)) / ln n
// (math_core/cuda_kernels.py:280; math_core/cpu_kernels.py:249).
__device__ __forceinline__ SampleOut escaped_sample(int k, double mag2, double inv_ln) {
    SampleOut o;
    const double log_mag = log(mag2);
    o.k = k;
    o.glitch = 0;
    o.iters = k;
    o.leaps = 0;
    o.iters2 = 0;
    if (log_mag > 1.0) {
        const double nu = (log(0.5 * log_mag) - kLnBailoutLog) * inv_ln;
        o.s = __fsub_rn((float)((double)k + 1.0), (float)nu);
        o.s64 = ((double)k + 1.0) - nu;
    } else {
        o.s = (float)k;
        o.s64 = (double)k;
    }
    return o;
}

// 1/ln(n) rounded through float32 for Multibrot, else 1/ln 2.
__host__ __device__ __forceinline__ double inv_ln_for(int fractal_type, int gen_n) {
    if (fractal_type == 4 && gen_n > 1) return (double)(float)(1.0 / log((double)gen_n));
    return kInvLn2;
}

// Steps of a span: consecutive steps of a packed orbit that the coarse kernels take without a
// test where the delta lies in the window stored in the record (orbit_window, ap_pack.cu).
constexpr int kSpan = 8;

// 2 a + b: doubling is exact, so the fused form rounds once where the two operations do, to the same
// value.  The perturbation steps, which write 2 Z + dz and 2 (...) + dc, are bound by the FP64 pipe: a
// Mandelbrot step of the CPU profile is 11 operations instead of 14 (1279x719 at 1e-26 with a series,
// a frame 1937 -> 1807 us).
__device__ __forceinline__ double twice_plus(double a, double b) { return fma(2.0, a, b); }

// ---------------------------------------------------------------- colouring
// Transfer functions of math_core/cuda_kernels.py:157-259, evaluated in
// float64 on the float32 smooth value.

// Python's x % M for M = 1, 2.  fmod is exact, and so is x - M trunc(x / M) here: x / M only moves the
// exponent, the multiple of M is exact, and the difference is representable (it is the fmod).
template <int M>
__device__ __forceinline__ double py_mod(double x) {
    const double m = (double)M;
    double r = M == 2 ? x - 2.0 * trunc(0.5 * x) : x - trunc(x);
    if (r != 0.0) {
        if (r < 0.0) r += m;
    } else {
        r = 0.0;
    }
    return r;
}

__device__ __forceinline__ double tri_wave(double phase) {
    return 1.0 - fabs((phase < 0.0 ? phase + 2.0 : phase) - 1.0);
}

// sqrt of the smooth value: the CPU reference holds it as float32 and Numba
// evaluates math.sqrt(float32) in float32; the CUDA reference holds float64.
__device__ __forceinline__ double sqrt_s(double s, bool f32) {
    return f32 ? (double)__fsqrt_rn((float)s) : sqrt(s);
}

// What a transfer function takes from the frame alone: computed once per block or thread (a tanh,
// an exp or a division each) instead of once per sample.
struct Palette {
    double dens, cont, off, off2, m, k, scale;
};

constexpr double kTwoPi = 6.28318530718;

// hist: the histogram transfer (scheme 11), where m is 1 / max(1, max_iter).
__device__ __forceinline__ Palette palette_of(const ApFrameParams& p, bool hist) {
    Palette c;
    c.dens = p.color_density <= 0.0 ? 1.0 : p.color_density;
    c.cont = p.color_contrast <= 0.0 ? 1.0 : p.color_contrast;
    c.off = p.palette_offset;
    c.off2 = c.off * 2.0;
    c.m = c.k = c.scale = 0.0;
    if (hist) {
        c.m = 1.0 / fmax(1.0, (double)p.max_iter);
        return c;
    }
    switch (p.scheme_id) {
    case 1: c.m = 0.45 * c.dens; break;
    case 2: {
        c.m = 0.125 * c.dens;
        c.k = 4.0 * c.cont;
        const double td = tanh(0.5 * c.k);
        c.scale = fabs(td) > 1e-7 ? 0.5 / td : 0.5186574;
        break;
    }
    case 3: {
        c.m = 0.125 * c.dens;
        c.k = 3.0 * c.cont;
        const double ed = exp(c.k) - 1.0;
        c.scale = fabs(ed) > 1e-7 ? 1.0 / ed : 0.0523957;
        break;
    }
    case 4: c.m = 0.5 * c.dens; break;
    case 5:
        c.m = 0.05 * c.dens;
        c.k = 1.61803398875 * c.cont;
        break;
    case 6: c.m = 0.08 * c.dens; break;
    case 7: {
        c.m = 0.05 * c.dens;
        const double b = 0.5 * c.cont;
        c.k = b;
        const double ns = 1.0 + b + b * b + b * b * b;
        c.scale = ns > 1e-7 ? 0.5 / ns : 0.26666666666666666;
        break;
    }
    case 8: c.m = 0.1 * c.dens; break;
    case 9:
        c.m = 0.04 * c.dens;
        c.k = 0.00008 * c.dens * c.cont;
        break;
    case 10: c.m = -0.06 * c.cont; break;
    default: c.m = 0.125 * c.dens;
    }
    return c;
}

__device__ __forceinline__ double palette_norm(const Palette& c, double s, int scheme, bool f32) {
    switch (scheme) {
    case 1: return tri_wave(py_mod<2>(log(s * c.cont + 1.0) * c.m + c.off2));
    case 2: {
        const double tri = tri_wave(py_mod<2>(sqrt_s(s, f32) * c.m + c.off2));
        return 0.5 + tanh((tri - 0.5) * c.k) * c.scale;
    }
    case 3: {
        const double tri = tri_wave(py_mod<2>(sqrt_s(s, f32) * c.m + c.off2));
        return (exp(c.k * tri) - 1.0) * c.scale;
    }
    case 5: {
        const double ang = s * c.m + c.off * kTwoPi;
        return 0.5 + 0.25 * (sin(ang) + sin(ang * c.k));
    }
    case 6: {
        const double ang = s * c.m + c.off * kTwoPi;
        const double val = 0.5 * (1.0 - cos(ang));
        return c.cont != 1.0 ? pow(val, c.cont) : val;
    }
    case 7: {
        const double ph = s * c.m + c.off * kTwoPi;
        const double b = c.k;
        const double wave = sin(ph) + b * sin(ph * 2.0 + 1.2) + (b * b) * sin(ph * 4.0 + 2.4) +
                            (b * b * b) * sin(ph * 8.0 + 3.6);
        return 0.5 + c.scale * wave;
    }
    case 8: {
        double tri = tri_wave(py_mod<2>(sqrt_s(s, f32) * c.m + c.off2));
        if (c.cont != 1.0) tri = pow(tri, c.cont);
        const double t2 = tri * tri;
        return t2 * tri * (tri * (tri * 6.0 - 15.0) + 10.0);
    }
    case 9: {
        const double ang = s * c.m + (s * s) * c.k + c.off * kTwoPi;
        return 0.5 + 0.5 * sin(ang);
    }
    case 10: {
        const double raw = py_mod<1>(1.0 - exp(c.m * sqrt(s * c.dens)) + c.off);
        return raw >= 0.0 ? raw : raw + 1.0;
    }
    default: {  // scheme 0, 4 and every id above 10
        const double tri = tri_wave(py_mod<2>(sqrt_s(s, f32) * c.m + c.off2));
        return c.cont != 1.0 ? pow(tri, c.cont) : tri;
    }
    }
}

// The same in one function for kernels that colour beside other work.
static __device__ __noinline__ double palette_norm_call(const Palette& c, double s, int scheme, bool f32) {
    return palette_norm(c, s, scheme, f32);
}

// Histogram-equalised transfer (math_core/cuda_kernels.py:237-259).
__device__ __forceinline__ double cdf_norm(const Palette& pc, double s, const float* __restrict__ cdf,
                                           int num_bins, double contrast) {
    if (s < 0.0) return -1.0;
    const double pos = (s * pc.m) * (double)(num_bins - 1);
    const int k = (int)pos;
    double c;
    if (k >= num_bins - 1) {
        c = (double)__ldg(cdf + num_bins - 1);
    } else if (k < 0) {
        c = (double)__ldg(cdf);
    } else {
        const double frac = pos - (double)k;
        const float c0 = __ldg(cdf + k), c1 = __ldg(cdf + k + 1);
        c = (double)c0 + frac * (double)__fsub_rn(c1, c0);
    }
    if (contrast != 1.0 && contrast > 0.0) c = pow(c, contrast);
    return tri_wave(py_mod<2>(c * (2.0 * pc.dens) + pc.off2));
}

// 2048-entry LUT lerp (math_core/cuda_kernels.py:157-168).
__device__ __forceinline__ void lut_lerp(const float* __restrict__ lut, double norm, double& r,
                                         double& g, double& b) {
    const double n = norm < 0.0 ? 0.0 : (norm > 1.0 ? 1.0 : norm);
    const double pos = n * 2047.0;
    const int i0 = (int)pos;
    const int i1 = i0 >= 2047 ? 2047 : i0 + 1;
    const double frac = pos - (double)i0;
    const double inv = 1.0 - frac;
    r = (double)__ldg(lut + i0 * 3 + 0) * inv + (double)__ldg(lut + i1 * 3 + 0) * frac;
    g = (double)__ldg(lut + i0 * 3 + 1) * inv + (double)__ldg(lut + i1 * 3 + 1) * frac;
    b = (double)__ldg(lut + i0 * 3 + 2) * inv + (double)__ldg(lut + i1 * 3 + 2) * frac;
}

// A colour component as its integer: int conversion where it is in range (LUT values are 0..65535),
// the 64-bit one of the reference's casts otherwise.
__device__ __forceinline__ unsigned colour_int(double v) {
    const double t = v + 0.5;
    return fabs(t) < 1073741824.0 ? (unsigned)(int)t : (unsigned)(long long)t;
}

__device__ __forceinline__ void store_rgb(void* rgb, int is_hdr, size_t idx, double r, double g,
                                          double b) {
    if (is_hdr) {
        uint16_t* o = static_cast<uint16_t*>(rgb) + idx * 3;
        o[0] = (uint16_t)colour_int(r);
        o[1] = (uint16_t)colour_int(g);
        o[2] = (uint16_t)colour_int(b);
    } else {
        uint8_t* o = static_cast<uint8_t*>(rgb) + idx * 3;
        o[0] = (uint8_t)colour_int(r);
        o[1] = (uint8_t)colour_int(g);
        o[2] = (uint8_t)colour_int(b);
    }
}

// Colour of one smooth value under the frame's transfer function (c = palette_of(p, hist)).
__device__ __forceinline__ void colour_of(const ApFrameParams& p, const Palette& c, const float* __restrict__ lut,
                                          const float* __restrict__ cdf, bool hist, double s,
                                          double& r, double& g, double& b) {
    const double norm = hist ? cdf_norm(c, s, cdf, p.num_bins, p.color_contrast)
                             : palette_norm_call(c, s, p.scheme_id, p.arith == AP_ARITH_REF_CPU);
    lut_lerp(lut, norm, r, g, b);
}

}  // namespace ap
