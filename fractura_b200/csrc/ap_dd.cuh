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

// Integer tests of the high words of the values that a run of steps has started from, off the FP64
// pipe and off the steps' dependent chain: every high part 0 or 2^-200 <= |v| < 181 (181^2 + 181^2 <
// 65536), every low part 0 or at least 2^-700.  What is below 2^-1042 counts as 0: its products can
// differ from the general step's in the last bit of a subnormal number, 2^-1074.
struct PlainRange {
    unsigned top = 0u, high = ~0u, low = ~0u;
    __device__ __forceinline__ void add(dd x, dd y) {
        const unsigned hx = (unsigned)__double2hiint(x.hi) & 0x7fffffffu, hy = (unsigned)__double2hiint(y.hi) & 0x7fffffffu;
        const unsigned lx = (unsigned)__double2hiint(x.lo) & 0x7fffffffu, ly = (unsigned)__double2hiint(y.lo) & 0x7fffffffu;
        top = max(top, max(hx, hy));
        high = min(high, min(hx - 1u, hy - 1u));  // 0 counts as the largest
        low = min(low, min(lx - 1u, ly - 1u));
    }
    static constexpr unsigned k181 = 0x4066a000u, kHigh = (1023u - 200u) << 20, kLow = (1023u - 700u) << 20;
    __device__ __forceinline__ bool plain() const {
        return (top < k181) & (high >= kHigh - 1u) & (low >= kLow - 1u);
    }
    // the same without 181, for a step whose |z|^2 is tested
    __device__ __forceinline__ bool finite() const {
        return (top < (1023u + 400u) << 20) & (high >= kHigh - 1u) & (low >= kLow - 1u);
    }
};

// One step z <- z^2 + c (SHIP: (|Re z| + i |Im z|)^2 - i-mirrored c) of the reference's operations
// in its order, for any operands; zx2, zy2 the squares.
template <int ARITH, bool SHIP>
__device__ __forceinline__ void dd_step_general(dd& zx, dd& zy, dd zx2, dd zy2, dd cx, dd cy) {
    const dd sub = dd_sub(zx2, zy2);
    const dd zxy = SHIP ? dd_mul<ARITH>(dd_abs(zx), dd_abs(zy)) : dd_mul<ARITH>(zx, zy);
    const dd two{zxy.hi * 2.0, zxy.lo * 2.0};
    zx = dd_add(sub, cx);
    zy = SHIP ? dd_sub(two, cy) : dd_add(two, cy);
}

// The same for normalised operands in PlainRange (see dd_quad_orbit).  Returns |z|^2 as the general
// step's test forms it.
template <bool SHIP>
__device__ __forceinline__ double dd_step_plain(dd& zx, dd& zy, dd cx, dd cy) {
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
    return zx2.hi + zy2.hi;
}

// The orbit of z under z^2 + c (SHIP: Burning Ship), bit for bit (but for the signs of zeros, which
// no magnitude depends on) as dd_step_general gives it in either profile, in 58 FP64 operations a
// step instead of 117 (REF_CPU, whose Dekker product takes 17) or 80 (REF_CUDA):
//   * Dekker's product error is exact, as fma(a, b, -ab) is, wherever no partial product
//     underflows, so both profiles take the two-operation product;
//   * every second sum of a normalised operation has its operands in order of magnitude
//     (add_normalised; a product's correction is below 2^-50 of it): 3 operations for 6;
//   * 2 z_x and 2 z_y are formed once for the squares' cross terms and for 2 z_x z_y
//     (scaling by 2 commutes with every rounding that does not underflow);
//   * while both high parts are below 181 the orbit cannot have passed the bailout, so |z|^2 goes
//     unformed in the blocks.  A z with a high part below 2^-200 or a low part below 2^-700 (not 0),
//     where a product could underflow, takes the general step.
// The first kDdLead steps are tested one by one: a shallow frame, whose pixels escape there, is bound by
// the FP64 pipe and would run up to two blocks for nothing (1280x720 Burning Ship at 1e-20, whose pixels
// escape after 26 steps: a frame 289 us with blocks from the first step on, 265 so).
// Then the steps run in blocks whose tests are gathered into three words; where they fail, the block is
// taken again from its start by tested steps, which the lanes of a warp do together.  With a test
// and a branch a step throughout, the chain of a lone warp waited for all four parts of z: a deep frame
// that leaves most of the GPU idle is bound by it (128x96 Mandelbrot at 1e-18, depth 8500, REF_CUDA:
// 1559 us with a test a step, 1230 with blocks and a flag, 1117 with the three words, 1140 with the first
// 32 steps tested; 1217 before the short step), a large one by the FP64 pipe (960x540 20.1 -> 15.5 ms, 16.2 with a test a step; 960x540
// Burning Ship at 2e-17, depth 6000, REF_CPU 13.1 -> 7.2 ms, 7.5 with a test a step).  Blocks of 4, 8 and
// 16 steps: 128x96 1117, 1117 and 1093 us; 599x400 Burning Ship at depth 6000 4246, 3954 and 3981.
constexpr int kDdBlock = 8, kDdLead = 32;
// Returns the escape step, or -1.
template <int ARITH, bool SHIP>
__device__ __forceinline__ int dd_quad_orbit(dd zx, dd zy, const dd cx, const dd cy, int max_iter,
                                             bool normalised, double& mag2_out) {
    int tested = kDdLead;
    for (int k = 0; k < max_iter; tested = kDdBlock) {
        for (const int stop = k + min(tested, max_iter - k); k < stop; ++k) {
            PlainRange range;
            range.add(zx, zy);
            double mag2;
            if (normalised && range.finite()) {
                mag2 = dd_step_plain<SHIP>(zx, zy, cx, cy);
            } else {
                const dd zx2 = dd_sqr<ARITH>(zx), zy2 = dd_sqr<ARITH>(zy);
                mag2 = zx2.hi + zy2.hi;
                dd_step_general<ARITH, SHIP>(zx, zy, zx2, zy2, cx, cy);
            }
            if (mag2 > kBailout) {
                mag2_out = mag2;
                return k;
            }
        }
        while (normalised && max_iter - k >= kDdBlock) {
            const dd bx = zx, by = zy;
            PlainRange range;
#pragma unroll
            for (int t = 0; t < kDdBlock; ++t) {
                range.add(zx, zy);
                dd_step_plain<SHIP>(zx, zy, cx, cy);
            }
            if (!range.plain()) {
                zx = bx;
                zy = by;
                break;
            }
            k += kDdBlock;
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
