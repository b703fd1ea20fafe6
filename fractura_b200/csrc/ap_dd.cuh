// ap_dd.cuh -- double-double direct iteration.
//
// Semantics of compute_dd_sample (math_core/cuda_kernels.py:321-418) and
// cpu_compute_dd_sample (math_core/cpu_kernels.py:271-369).  The two
// references differ only in the error-free product: the CUDA build uses
// fma(a, b, -a*b), the CPU build a Dekker split; ARITH selects which.
#pragma once

#include "ap_common.cuh"

namespace ap {

struct dd {
    double hi, lo;
};

__device__ __forceinline__ dd two_sum(double a, double b) {
    const double s = a + b;
    const double v = s - a;
    const double e = (a - (s - v)) + (b - v);
    return {s, e};
}

template <int ARITH>
__device__ __forceinline__ dd two_prod(double a, double b) {
    if constexpr (ARITH == AP_ARITH_REF_CPU) {
        // Dekker split with 2^27 + 1 (math_core/cpu_kernels.py:104-113).
        double c = 134217729.0 * a;
        const double a_hi = c - (c - a);
        const double a_lo = a - a_hi;
        c = 134217729.0 * b;
        const double b_hi = c - (c - b);
        const double b_lo = b - b_hi;
        const double p = a * b;
        const double e = ((a_hi * b_hi - p) + a_hi * b_lo + a_lo * b_hi) + a_lo * b_lo;
        return {p, e};
    } else {
        const double p = a * b;
        return {p, fma(a, b, -p)};
    }
}

__device__ __forceinline__ dd dd_abs(dd a) {
    return (a.hi < 0.0 || (a.hi == 0.0 && a.lo < 0.0)) ? dd{-a.hi, -a.lo} : a;
}

__device__ __forceinline__ dd dd_add(dd a, dd b) {
    const dd s = two_sum(a.hi, b.hi);
    return two_sum(s.hi, s.lo + a.lo + b.lo);
}

__device__ __forceinline__ dd dd_sub(dd a, dd b) {
    const dd s = two_sum(a.hi, -b.hi);
    return two_sum(s.hi, s.lo + a.lo - b.lo);
}

template <int ARITH>
__device__ __forceinline__ dd dd_mul(dd a, dd b) {
    const dd p = two_prod<ARITH>(a.hi, b.hi);
    return two_sum(p.hi, p.lo + a.hi * b.lo + a.lo * b.hi);
}

template <int ARITH>
__device__ __forceinline__ dd dd_mul_f64(dd a, double b) {
    const dd p = two_prod<ARITH>(a.hi, b);
    return two_sum(p.hi, p.lo + a.lo * b);
}

template <int ARITH>
__device__ __forceinline__ dd dd_sqr(dd a) {
    const dd p = two_prod<ARITH>(a.hi, a.hi);
    return two_sum(p.hi, p.lo + 2.0 * a.hi * a.lo);
}

// s = a + b and its error for b = 0 or a's exponent at least b's (Dekker's quick sum): the
// values of two_sum(a, b) in 3 operations instead of 6.
__device__ __forceinline__ dd quick_sum(double a, double b) {
    const double s = a + b;
    return {s, b - (s - a)};
}

// dd_add of normalised operands (|lo| at most half an ulp of hi).  The second sum is quick:
// where the first one is inexact it cancels at most one bit and the low parts are far
// below it; where it is exact and not zero it is a multiple of the smaller operand's ulp w,
// and the low parts add up to at most w (equal exponents) or 3/4 ulp of the larger operand
// (exponents one apart, s a multiple of half that ulp), so their exponent is not above s's;
// a zero sum leaves an exact quick sum.
__device__ __forceinline__ dd add_normalised(dd a, dd b) {
    const dd s = two_sum(a.hi, b.hi);
    return quick_sum(s.hi, s.lo + a.lo + b.lo);
}

__device__ __forceinline__ bool dd_normalised(dd a) { return a.hi + a.lo == a.hi; }

// Integer tests of a high word, off the FP64 pipe.  plain_high: 2^-200 <= |v| < 181
// (181^2 + 181^2 < 65536); zero is not plain.  plain_low: |v| >= 2^-700, or 0.
__device__ __forceinline__ bool plain_high(double v) {
    constexpr unsigned lo = (1023u - 200u) << 20, hi = 0x4066a000u;  // the high words of 2^-200 and 181.0
    return ((unsigned)__double2hiint(v) & 0x7fffffffu) - lo < hi - lo;
}
__device__ __forceinline__ bool plain_low(double v) {
    const unsigned h = (unsigned)__double2hiint(v) & 0x7fffffffu;
    return h >= (1023u - 700u) << 20 || (h | (unsigned)__double2loint(v)) == 0u;
}

// One step z <- z^2 + c (SHIP: (|Re z| + i |Im z|)^2 - i-mirrored c) of the reference's
// operations in its order, for any operands.
struct dd2 {
    dd x, y;
};
template <int ARITH, bool SHIP>
__device__ __noinline__ dd2 dd_step_general(dd2 z, dd2 c) {
    const dd sub = dd_sub(dd_sqr<ARITH>(z.x), dd_sqr<ARITH>(z.y));
    const dd zxy = SHIP ? dd_mul<ARITH>(dd_abs(z.x), dd_abs(z.y)) : dd_mul<ARITH>(z.x, z.y);
    const dd two{zxy.hi * 2.0, zxy.lo * 2.0};
    return {dd_add(sub, c.x), SHIP ? dd_sub(two, c.y) : dd_add(two, c.y)};
}

// The orbit of z under z^2 + c (SHIP: Burning Ship), bit for bit as dd_step_general gives it
// in either profile, in 58 FP64 operations a step instead of 117 (REF_CPU, whose Dekker
// product takes 17) or 80 (REF_CUDA):
//   * Dekker's product error is exact, as fma(a, b, -ab) is, wherever no partial product
//     underflows, so both profiles take the two-operation product;
//   * every second sum of a normalised operation has its operands in order of magnitude
//     (add_normalised; a product's correction is below 2^-50 of it): 3 operations for 6;
//   * 2 z_x and 2 z_y are formed once for the squares' cross terms and for 2 z_x z_y
//     (scaling by 2 commutes with every rounding that does not underflow);
//   * while both high parts are below 181 the orbit cannot have passed the bailout, so |z|^2
//     is formed only by the general step, which every other z takes: one near the bailout,
//     and one with a high part below 2^-200 (zero included: the first step) or a low part
//     below 2^-700, where a product could underflow.
// Bound by the FP64 pipe (84 % of its issue slots; 59.5 FP64 instructions a step and warp).
// Measured: 1280x720 Burning Ship at 2e-17, max_iter 20000, 2x SSAA, REF_CPU 102.0 -> 56.6 ms;
// 960x540 Mandelbrot at 1e-18, REF_CUDA 20.4 -> 16.6 ms.
// Returns the escape step, or -1.
template <int ARITH, bool SHIP>
__device__ __forceinline__ int dd_quad_orbit(dd zx, dd zy, const dd cx, const dd cy, int max_iter,
                                             bool normalised, double& mag2_out) {
    for (int k = 0; k < max_iter; ++k) {
        if (!(normalised && plain_high(zx.hi) && plain_high(zy.hi) && plain_low(zx.lo) && plain_low(zy.lo))) {
            const double mag2 = dd_sqr<ARITH>(zx).hi + dd_sqr<ARITH>(zy).hi;
            if (mag2 > kBailout) {
                mag2_out = mag2;
                return k;
            }
            const dd2 n = dd_step_general<ARITH, SHIP>(dd2{zx, zy}, dd2{cx, cy});
            zx = n.x;
            zy = n.y;
            continue;
        }
        const double x2 = zx.hi + zx.hi, y2 = zy.hi + zy.hi;
        double p = zx.hi * zx.hi;
        const dd zx2 = quick_sum(p, fma(zx.hi, zx.hi, -p) + x2 * zx.lo);
        p = zy.hi * zy.hi;
        const dd zy2 = quick_sum(p, fma(zy.hi, zy.hi, -p) + y2 * zy.lo);
        p = x2 * zy.hi;
        dd zxy = quick_sum(p, fma(x2, zy.hi, -p) + x2 * zy.lo + zx.lo * y2);  // 2 z_x z_y
        zx = add_normalised(add_normalised(zx2, dd{-zy2.hi, -zy2.lo}), cx);
        if (SHIP) {
            // 2 |z_x| |z_y|: the low part's sign turns with the high part's
            const int flip = __double2hiint(zxy.hi) & 0x80000000;
            zxy.hi = fabs(zxy.hi);
            zxy.lo = __hiloint2double(__double2hiint(zxy.lo) ^ flip, __double2loint(zxy.lo));
            zy = add_normalised(zxy, dd{-cy.hi, -cy.lo});
        } else {
            zy = add_normalised(zxy, cy);
        }
    }
    return -1;
}

template <int ARITH, bool MULTI>
__device__ __forceinline__ SampleOut dd_sample(dd cxv, dd cyv, const ApFrameParams& p) {
    const int ft = p.fractal_type;
    const int max_iter = p.max_iter;
    if (ft == 0) {
        const double xm = cxv.hi - 0.25;
        const double y2 = cyv.hi * cyv.hi;
        const double q = xm * xm + y2;
        if ((q * (q + xm) <= 0.25 * y2) || ((cxv.hi + 1.0) * (cxv.hi + 1.0) + y2 <= 0.0625))
            return skipped_sample();
    }
    const dd jx{p.julia_cx_hi, p.julia_cx_lo}, jy{p.julia_cy_hi, p.julia_cy_lo};
    dd zx, zy, cx, cy;
    if (ft == 2 || ft == 3) {
        zx = cxv; zy = cyv; cx = jx; cy = jy;
    } else {
        zx = {0.0, 0.0}; zy = {0.0, 0.0}; cx = cxv; cy = cyv;
    }
    if (!MULTI && ft >= 0 && ft <= 3) {
        const bool normalised = dd_normalised(zx) && dd_normalised(zy) && dd_normalised(cx) && dd_normalised(cy);
        double mag2 = 0.0;
        const int k = (ft & 1) ? dd_quad_orbit<ARITH, true>(zx, zy, cx, cy, max_iter, normalised, mag2)
                               : dd_quad_orbit<ARITH, false>(zx, zy, cx, cy, max_iter, normalised, mag2);
        return k < 0 ? interior_after(max_iter) : escaped_sample(k, mag2, kInvLn2);
    }
    if (MULTI && ft == 4) {
        const int n = p.gen_n;
        const double kr = p.gen_kr, ki = p.gen_ki;
        const double inv_ln = inv_ln_for(4, n);
        for (int k = 0; k < max_iter; ++k) {
            const dd zx2 = dd_sqr<ARITH>(zx), zy2 = dd_sqr<ARITH>(zy);
            const double mag2 = zx2.hi + zy2.hi;
            if (mag2 > kBailout) return escaped_sample(k, mag2, inv_ln);
            dd cr = zx, ci = zy;
            for (int t = 0; t < n - 1; ++t) {
                const dd re = dd_sub(dd_mul<ARITH>(cr, zx), dd_mul<ARITH>(ci, zy));
                const dd im = dd_add(dd_mul<ARITH>(cr, zy), dd_mul<ARITH>(ci, zx));
                cr = re;
                ci = im;
            }
            const dd kz_r = dd_sub(dd_mul_f64<ARITH>(zx, kr), dd_mul_f64<ARITH>(zy, ki));
            const dd kz_i = dd_add(dd_mul_f64<ARITH>(zy, kr), dd_mul_f64<ARITH>(zx, ki));
            zx = dd_add(dd_add(cr, kz_r), cx);
            zy = dd_add(dd_add(ci, kz_i), cy);
        }
        return interior_after(max_iter);
    }
    return interior_sample();
}

// Sub-sample -> DD coordinate (math_core/cuda_kernels.py:1685-1691, :1712-1719).
// MULTI: Multibrot (its power loop wants registers that the quadratic formulas can do without).
template <int ARITH, bool MULTI>
__device__ __forceinline__ SampleOut dd_sample_at(const ApFrameParams& p, double sub_i,
                                                  double sub_j) {
    const dd jdy = dd_mul_f64<ARITH>(dd{p.dy_hi, p.dy_lo}, sub_j);
    const dd cy = dd_sub(dd{p.y_max_hi, p.y_max_lo}, jdy);
    const dd idx = dd_mul_f64<ARITH>(dd{p.dx_hi, p.dx_lo}, sub_i);
    const dd cx = dd_add(dd{p.x_min_hi, p.x_min_lo}, idx);
    return dd_sample<ARITH, MULTI>(cx, cy, p);
}

}  // namespace ap
