// ap_fp64.cuh -- direct FP64 escape-time iteration for the five formulas.
//
// Semantics of compute_fp64_sample (math_core/cuda_kernels.py:264-317) and
// cpu_compute_fp64_sample (math_core/cpu_kernels.py:228-266).  ARITH picks
// which multiply-adds are fused:
//   AP_ARITH_REF_CPU  the fused/reassociated forms the reference's Numba CPU
//                     build executes (bit-identical to its output);
//   AP_ARITH_REF_CUDA the reference's CUDA source expressions, unfused.
#pragma once

#include "ap_common.cuh"

namespace ap {

constexpr int kKindQuad = 0, kKindShip = 1, kKindMulti = 4;

// Calls f with the Multibrot degree as a compile-time constant for 2..5, else with 0; for the
// quadratic kinds with 1 where fp64_step may fuse the doubling (`doubles`), else with 0.
template <int N>
struct Degree {
    __host__ __device__ constexpr int operator()() const { return N; }
};
template <typename F>
__device__ __forceinline__ void for_degree(int kind, int n, bool doubles, F&& f) {
    if (kind != kKindMulti) {
        if (doubles) f(Degree<1>());
        else f(Degree<0>());
        return;
    }
    switch (n) {
    case 2: f(Degree<2>()); break;
    case 3: f(Degree<3>()); break;
    case 4: f(Degree<4>()); break;
    case 5: f(Degree<5>()); break;
    default: f(Degree<0>());
    }
}

// Whether fma(2, zx zy, cy) is (2 zx) zy + cy in every step from zy on, so that a quadratic step of the
// CUDA profile is six FP64 operations instead of seven.  The two products differ only below the
// smallest normal number, 2^-1022, where the sum with |cy| >= 2^-960 is cy for both; and they are zeros
// of one sign throughout where cy = zy = 0.  1283x721 Julia with 2x SSAA 733 -> 681 us; second stages of
// perturbation (1279x719 at 1e-26 with a series, a frame) 1810 -> 1752 us.
__device__ __forceinline__ bool fp64_doubles(double zy, double cy) {
    return fabs(cy) >= 0x1p-960 || (cy == 0.0 && zy == 0.0);
}

// One step of z in the profile's roundings; zx2, zy2 the squares (quadratic kinds).  N: the
// Multibrot degree where it is known at compile time (2..5, the powers unrolled), else 0; for the
// quadratic kinds 1 where fp64_doubles holds, else 0.
template <int ARITH, int KIND, int N>
__device__ __forceinline__ void fp64_step(double& zx, double& zy, double zx2, double zy2, double cx, double cy,
                                          int n, double kr, double ki) {
    constexpr bool kCpu = (ARITH == AP_ARITH_REF_CPU);
    if (KIND == kKindQuad) {
        if (kCpu) {
            const double nzy = fma(zy + zy, zx, cy);
            zx = (cx - zy2) + zx2;
            zy = nzy;
        } else {
            zy = N == 1 ? twice_plus(zx * zy, cy) : 2.0 * zx * zy + cy;
            zx = zx2 - zy2 + cx;
        }
    } else if (KIND == kKindShip) {
        const double ax = fabs(zx), ay = fabs(zy);
        if (kCpu) {
            const double nzy = fma(ax, ay + ay, -cy);
            zx = (cx + zx2) - zy2;
            zy = nzy;
        } else {
            zy = N == 1 ? twice_plus(ax * ay, -cy) : 2.0 * ax * ay - cy;
            zx = zx2 - zy2 + cx;
        }
    } else {
        double zr = zx, zi = zy;
        const int powers = (N > 0 ? N : n) - 1;
#pragma unroll
        for (int t = 0; t < powers; ++t) {
            double nr, ni;
            if (kCpu) {
                nr = fma(zr, zx, -(zi * zy));
                ni = fma(zi, zx, zr * zy);
            } else {
                nr = zr * zx - zi * zy;
                ni = zr * zy + zi * zx;
            }
            zr = nr;
            zi = ni;
        }
        if (kCpu) {
            const double a = fma(zx, kr, -fma(ki, zy, -cx));
            const double b = fma(ki, zx, fma(zy, kr, cy));
            zx = a + zr;
            zy = b + zi;
        } else {
            const double kz_r = kr * zx - ki * zy;
            const double kz_i = kr * zy + ki * zx;
            zx = zr + kz_r + cx;
            zy = zi + kz_i + cy;
        }
    }
}

// |z|^2 as the profile forms it for the escape test.
template <int ARITH, int KIND>
__device__ __forceinline__ double fp64_mag2(double zx, double zy) {
    if (KIND == kKindMulti && ARITH == AP_ARITH_REF_CPU) return fma(zx, zx, zy * zy);
    return zx * zx + zy * zy;
}

// Steps tested one by one before the first block, and steps of a block.  Blocks of 8 took a
// 1283x721 Julia frame with 2x SSAA 772 us, blocks of 16 take 726; leads of 4, 8 and 16 time alike.
constexpr int kLead = 8;
constexpr int kBlock = 16;

// Whether an orbit that has passed the bailout keeps growing (see fp64_orbit).
__device__ __forceinline__ bool fp64_growing(int kind, double cx, double cy, int n, double kr, double ki) {
    return fabs(cx) <= 1000.0 && fabs(cy) <= 1000.0 &&
           (kind != kKindMulti || (n >= 2 && fabs(kr) <= 100.0 && fabs(ki) <= 100.0));
}

// The orbit of z: escape step and |z|^2 as testing every step gives them.  A step's test is on the
// step's dependent chain (square, add, compare, branch) and takes two of its FP64 operations, so
// after kLead tested steps (where most of a frame's pixels escape) the orbit runs in blocks of
// kBlock steps tested at the end only:
//   * once the computed |z|^2 has passed the bailout, 65536, every later one has too or is not a
//     number (`growing`: |c| <= 1415, and for Multibrot n >= 2 and |k| <= 142, so that
//     |f(z)| >= |z| (|z| - |k|) - |c| > 256 for |z| >= 256); a block that ends above it, or in
//     NaN, is run again step by step;
//   * a block that ends in the z that an earlier block ended in repeats from there for ever:
//     the pixel never escapes (Brent's search: the z compared with is renewed after 1, 2,
//     4, ... blocks; -0 equals 0 here, which no later magnitude depends on).
// Measured: 128x72 probe at depth 4000 147 -> 98 us a call (a single chain of three dependent
// operations a step), Julia 1283x721 with 2x SSAA 952 -> 726 us, 1920x1080 Multibrot n = 3 at depth
// 5000, whose bounded pixels repeat after about 470 steps, 5.27 -> 0.93 ms.
// Returns the escape step, or -1; `steps`: the iterations run.
template <int ARITH, int KIND, int N>
__device__ __forceinline__ int fp64_orbit(double zx, double zy, double cx, double cy, int max_iter, bool growing,
                                          int n, double kr, double ki, double& mag2_out, int& steps) {
    int k = 0;
    int stop = growing && max_iter > kLead + kBlock ? kLead : max_iter;  // the tested steps: k in [k, stop)
    for (;;) {
        for (; k < stop; ++k) {
            double zx2 = 0.0, zy2 = 0.0, mag2;
            if (KIND == kKindMulti) {
                mag2 = fp64_mag2<ARITH, KIND>(zx, zy);
            } else {
                zx2 = zx * zx;
                zy2 = zy * zy;
                mag2 = zx2 + zy2;
            }
            if (mag2 > kBailout) {
                mag2_out = mag2;
                steps = k;
                return k;
            }
            fp64_step<ARITH, KIND, N>(zx, zy, zx2, zy2, cx, cy, n, kr, ki);
        }
        if (stop == max_iter) break;
        stop = max_iter;
        const bool doubles = ARITH != AP_ARITH_REF_CPU && fp64_doubles(zy, cy);
        double sx = zx, sy = zy;  // the z that block ends are compared with
        int left = 1, window = 1;
        while (max_iter - k >= kBlock) {
            const double bx = zx, by = zy;
            auto block = [&](auto form) {
#pragma unroll
                for (int t = 0; t < kBlock; ++t)
                    fp64_step<ARITH, KIND, form()>(zx, zy, zx * zx, zy * zy, cx, cy, n, kr, ki);
            };
            if (KIND != kKindMulti && doubles) block(Degree<1>());
            else block(Degree<N>());
            if (!(fp64_mag2<ARITH, KIND>(zx, zy) <= kBailout)) {
                zx = bx;
                zy = by;
                break;
            }
            k += kBlock;
            if (zx == sx && zy == sy) {
                steps = k;
                return -1;
            }
            if (--left == 0) {
                sx = zx;
                sy = zy;
                window *= 2;
                left = window;
            }
        }
    }
    steps = max_iter;
    return -1;
}

template <int ARITH>
__device__ __forceinline__ SampleOut fp64_sample(double x, double y, const ApFrameParams& p) {
    constexpr bool kCpu = (ARITH == AP_ARITH_REF_CPU);
    const int ft = p.fractal_type;

    if (ft == 0) {
        // Main cardioid and period-2 bulb early-out.
        const double xm = x - 0.25;
        const double y2 = y * y;
        const double q = kCpu ? fma(xm, xm, y2) : xm * xm + y2;
        const double xp = x + 1.0;
        const double b = kCpu ? fma(xp, xp, y2) : xp * xp + y2;
        if ((q * (q + xm) <= 0.25 * y2) || (b <= 0.0625)) return skipped_sample();
    }
    if (ft < 0 || ft > 4) return interior_sample();
    const bool julia = ft == 2 || ft == 3;
    const double zx = julia ? x : 0.0, zy = julia ? y : 0.0;
    const double cx = julia ? p.julia_cx_hi : x, cy = julia ? p.julia_cy_hi : y;
    const int n = p.gen_n;
    const double kr = p.gen_kr, ki = p.gen_ki;
    const bool growing = fp64_growing(ft == 4 ? kKindMulti : kKindQuad, cx, cy, n, kr, ki);
    double mag2 = 0.0;
    int steps = 0, k;
    if (ft == 4) {
        for_degree(kKindMulti, n, false, [&](auto degree) {
            k = fp64_orbit<ARITH, kKindMulti, degree()>(zx, zy, cx, cy, p.max_iter, growing, n, kr, ki, mag2, steps);
        });
    } else if (ft & 1) {
        k = fp64_orbit<ARITH, kKindShip, 0>(zx, zy, cx, cy, p.max_iter, growing, n, kr, ki, mag2, steps);
    } else {
        k = fp64_orbit<ARITH, kKindQuad, 0>(zx, zy, cx, cy, p.max_iter, growing, n, kr, ki, mag2, steps);
    }
    if (k >= 0) return escaped_sample(k, mag2, inv_ln_for(ft, n));
    return interior_after(steps);
}

}  // namespace ap
