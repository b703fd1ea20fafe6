// ap_coarse.cuh -- one pixel of a coarse FP64-delta perturbation pass on packed inputs.
//
// Same results as the generic render pass (ap_perturb.cuh) for tier
// AP_TIER_PERTURB in AP_MODE_COARSE without in-kernel colouring; it is picked
// by ap_render_pass when the buffers carry the packed orbit (ap_pack_orbit)
// and, with BLA, the packed table (ap_pack_bla).  What changes is only how the
// loop gets its inputs:
//   * one 32-byte record per step: Z_k, a safe radius (its low word: the span window) and the
//     level-0 BLA radius.  While |dz| is below the safe radius neither the escape test nor
//     the Pauldelbrot test can fire, so |Z + dz|^2 and the threshold are not
//     formed (the rounded |dz|^2 decides, and the BLA test reuses it);
//   * runs of plain steps of z^2 + c without a test each (span_steps), stage 2 in blocks tested at
//     their end, and whole cycles of bounded pixels added at once (cycle_visit);
//   * the 16 BLA radii of step k in one 128-byte row.  Radii never increase
//     with the level (each level's radius is the min of its first half's), and
//     levels past the end of the orbit hold 0, so the largest admissible level
//     -- the reference's top-down scan -- is a count, taken in two rounds of three loads;
//   * formula, BLA presence and arithmetic profile are template parameters;
//   * no colouring (ap_colour runs afterwards), keeping registers low.
#pragma once

#include <climits>

#include "ap_common.cuh"
#include "ap_fp64.cuh"

namespace ap {

constexpr int kFtQuad = 0;   // Mandelbrot (0) and its Julia set (2)
constexpr int kFtShip = 1;   // Burning Ship (1) and its Julia set (3)
constexpr int kFtMulti = 4;  // Multibrot z^n + k z + c

// Calls power() n - 1 times, the common degrees unrolled: the same operations in the
// same order, and what the last call prepares for a next one is dead and goes.
template <typename F>
__device__ __forceinline__ void for_powers(int n, F&& power) {
    switch (n) {
    case 2: power(); break;
    case 3: power(); power(); break;
    case 4: power(); power(); power(); break;
    case 5: power(); power(); power(); power(); break;
    default:
        for (int t = 0; t < n - 1; ++t) power();
    }
}

// |Z + dz| - |Z| of one component, given z = Z + dz and a = 2 Z + dz (each rounded): the
// reference's s dz where z keeps the sign s of Z and -s a where it does not.  s is Z's sign bit,
// so the test and the products by s = +-1 are integer operations on the high words (they were
// 5 of the 12 FP64-pipe operations a component took).  z = 0 passes for either sign: then
// dz = -Z and a = Z, and both forms give s dz.
__device__ __forceinline__ double fold_delta(double Z, double z, double dz, double a) {
    const int s = __double2hiint(Z);
    const double v = (__double2hiint(z) ^ s) >= 0 ? dz : -a;
    return __hiloint2double(__double2hiint(v) ^ (s & 0x80000000), __double2loint(v));
}

// 32-byte record through the read-only path, as two 128-bit loads: the loops wait for it, and one
// 256-bit load takes 58 cycles where these take 40 (1920x1080 at 1e-26, one-pass rebasing with leaps,
// 19.9 -> 19.4 ms; at 1e-160 without leaps 10.4 -> 9.7).
__device__ __forceinline__ double4 ldg4(const double4* p) {
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldg(q), c = __ldg(q + 1);
    return make_double4(a.x, a.y, c.x, c.y);
}

// Cycle detection.  A bounded pixel mostly settles on an exact cycle: its state returns bit for
// bit, and everything between the two visits repeats until max_iter.  The iterations of whole
// further cycles are then added at once.  The states compared are
//   * the delta at a restart (one-pass rebasing: m = 0, so the delta is the whole state);
//   * the delta at a step of the reference's periodic tail (a bounded reference that settled on
//     a cycle of its own: Z_{m+p} = Z_m bit for bit from m = s0 on, found by ap_pack_orbit),
//     against one at the same phase of the tail: with no restart in between, or at the same m.
// Brent's search: each visited state is compared with one kept state, and the kept one is renewed
// at visits 1, 2, 4, ...  Every fourth restart is visited (every 32nd of the Burning Ship), from the
// kFirstRestart-th on (escaping pixels have few), and the tail every kTailStride steps: a cycle is
// found as some whole number of its turns.
// What bounds the repetition: leaps are capped so that k stays within max_iter and m + 2^d below
// the orbit's end, where the radii of longer levels are 0.  A cycle of dk iterations holds no
// leap longer than what remains of it, so each repetition that ends by max_iter (and, in the
// tail, below the orbit's end) takes the same leaps; what is left after those runs as always.
// -0 and 0 compare equal: no later magnitude depends on the sign of a zero.
// Measured: 21 mixed tiles in one batch launch 187.6 -> 40.1 ms (bounded pixels were 96-99 % of
// the iterations of the Multibrot tiles and settle after 1000-14000 steps; of max_iter 20000-90000).
// The kept state, 28 bytes a pixel, is touched rarely.  The per-frame kernel keeps it in local memory
// (volatile: not in registers): in shared memory it took L1 capacity from the records and rows, which
// decide where the orbit is long (1920x1080 at 1e-26, 30000 records, leaps of tolerance 1e-5, one-pass
// rebasing 6.23 -> 5.70 ms).  The batch kernel, whose slots move, keeps it in shared memory beside them.
template <int N>
struct CycleStore {
    double x[N], y[N];
    int k[N], m[N], visits[N];
};
struct CycleLocal {
    volatile double x[1], y[1];
    volatile int k[1], m[1], visits[1];
};
constexpr int kTailStride = 64;
constexpr int kFirstRestart = 16;

// The reference's tail: period p (0: none) from step s0 on, as ap_pack_orbit leaves it in the
// last record's fourth slot (-(4096 s0 + p); no radius is negative, so no leap reads it as one),
// where it holds at least two periods and 64 steps.
struct OrbitTail {
    int p, s0;
};
__device__ __forceinline__ OrbitTail orbit_tail(const double4* __restrict__ orb, int ref_len) {
    const double t = -__ldg(reinterpret_cast<const double*>(orb + ref_len) + 3);
    if (!(t > 0.0)) return {0, INT_MAX};
    const int s0 = (int)(t * (1.0 / 4096.0)), p = (int)(t - 4096.0 * (double)s0);
    if (ref_len - 1 - s0 < max(2 * p, 64)) return {0, INT_MAX};
    return {p, s0};
}
__device__ __forceinline__ bool has_tail(const double4* __restrict__ orb, int ref_len) {
    return orbit_tail(orb, ref_len).p > 0;
}

// A visit of state (x, y) at k iterations and reference index m (0: a restart; else a tail step
// at the kept state's phase).  Returns the length of the cycle closed, 0 when none is.
template <class Store>
__device__ __forceinline__ int cycle_visit(Store& C, int q, double x, double y, int k, int m) {
    const int visits = C.visits[q];
    if (visits > 0 && C.x[q] == x && C.y[q] == y) {
        const int km = C.k[q], mm = C.m[q];  // m = -1: z itself, past the reference (stage 2)
        if (m == mm || (m > 0 && mm > 0 && m - mm == k - km)) return k - km;
    }
    if ((visits & (visits - 1)) == 0) {
        C.x[q] = x;
        C.y[q] = y;
        C.k[q] = k;
        C.m[q] = m;
    }
    C.visits[q] = visits + 1;
    return 0;
}

// Steps from tail step m to the next visit: to the kept state's phase, or (at_phase) past it.
template <class Store>
__device__ __forceinline__ int tail_gap(const Store& C, int q, OrbitTail tail, int m, bool at_phase) {
    if (at_phase) return ((kTailStride + tail.p - 1) / tail.p) * tail.p;
    if (C.visits[q] == 0 || C.m[q] == 0) return 0;
    const int d = (m - C.m[q]) % tail.p;
    return d == 0 ? 0 : (d < 0 ? -d : tail.p - d);
}

// A round of the batch kernel: it lasts until the SM's clock passes `end`, looked at every kRoundCheck
// loop iterations (`left`, the same for all lanes of a loop), and for the first iterations in any
// case.  Rounds counted in steps, weighted by formula, lasted as long as their block's dearest warp
// (21 mixed tiles 33.3 -> 29.2 ms with the clock; looking every 8, 16 or 32 iterations times alike).
constexpr int kRoundCheck = 16;
struct Round {
    int left;
    unsigned end;
    __device__ __forceinline__ bool over() {
        if (--left >= 0) return false;
        left = kRoundCheck - 1;
        return (int)((unsigned)clock() - end) >= 0;
    }
};

// One pixel of a coarse pass, resumable: pixel_begin sets it up, pixel_advance runs
// its stage-1 (perturbation) and stage-2 (direct) loops -- all of them, or until `round` is
// over when BUDGET is set, so that a persistent kernel can hand a lane whose pixel finished
// a new one -- and
// pixel_finish writes its outputs.  coarse_pixel runs the three in a row; the
// per-frame kernel below and the batch kernel (ap_batch.cu) share this code, so both
// give identical values.
struct PixelRun {
    double dzx, dzy;  // stage 1: the delta
    double zx, zy;    // stage 2: z itself
    double dcx, dcy;  // the pixel's offset from the reference
    int idx, k, k0, k2, glitch, leaps, skipped;
    int stage;        // 1 perturbation, 2 direct, 3 done
    int m, rebases;   // one-pass rebasing: reference index (k counts iterations), restarts
    SampleOut o;
};

template <int ARITH, int FT>
__device__ __forceinline__ bool pixel_begin(const ApFrameParams& p, const ApFrameBuffers& b, int i, int j,
                                            PixelRun& s) {
    s.idx = j * p.width + i;
    if (p.rebase_pass > 0 && b.glitch_in[s.idx] == 0) return false;
    const double sub_offset = ((double)p.factor - 1.0) * 0.5;
    const double sub_i = (double)(i * p.factor) + sub_offset;
    const double sub_j = (double)(j * p.factor) + sub_offset;
    s.dcy = (p.ref_py - sub_j) * p.dy_hi;
    s.dcx = (sub_i - p.ref_px) * p.dx_hi;
    const bool julia = (p.fractal_type == 2 || p.fractal_type == 3);
    s.dzx = julia ? s.dcx : 0.0;
    s.dzy = julia ? s.dcy : 0.0;
    s.k = 0;
    if (p.bbsa_skip > 0 && FT != kFtShip) {
        const double ux = s.dcx * p.bbsa_inv_r, uy = s.dcy * p.bbsa_inv_r;
        if (ux * ux + uy * uy <= 1.0) {
            bool eight = false;
            for (int q = 8; q < 16; ++q) eight |= (p.bbsa[q] != 0.0);
            const int top = eight ? 7 : 3;
            double tr = ux * p.bbsa[2 * top] - uy * p.bbsa[2 * top + 1];
            double ti = ux * p.bbsa[2 * top + 1] + uy * p.bbsa[2 * top];
            for (int q = top - 1; q >= 0; --q) {
                const double ar = p.bbsa[2 * q] + tr, ai = p.bbsa[2 * q + 1] + ti;
                tr = ux * ar - uy * ai;
                ti = ux * ai + uy * ar;
            }
            s.dzx = tr;
            s.dzy = ti;
            s.k = p.bbsa_skip;
        }
    }
    s.k0 = s.k;
    s.m = s.k;
    s.rebases = 0;
    s.k2 = -1;
    s.glitch = s.leaps = s.skipped = 0;
    s.stage = 1;
    s.o = interior_sample();
    return true;
}

// The largest admissible level of a leap: the levels whose radius covers |dz| are a prefix
// 0..lo (radii never increase with the level), so lo is a count.  Two rounds of three
// independent loads: the quarter of the row, then the level in it.
__device__ __forceinline__ int leap_level(const double* __restrict__ row, double dz_mag2, int hi) {
    int quarter = 0;
#pragma unroll
    for (int t = 1; t <= 3; ++t) quarter += (4 * t <= hi && dz_mag2 < __ldg(row + 4 * t)) ? 1 : 0;
    int lo = 4 * quarter;
#pragma unroll
    for (int t = 1; t <= 3; ++t) {
        const int d = 4 * quarter + t;
        lo += (d <= hi && dz_mag2 < __ldg(row + d)) ? 1 : 0;
    }
    return lo;
}

// Whether |dz|^2 (its high word) is not below a record's safe radius: unsigned words, so that a NaN of
// either sign (CUDA's own has the sign bit set) lies above every radius and a NaN delta is always
// tested -- the end of the reference is a radius of 0, which nothing passes untested.
__device__ __forceinline__ bool outside(int dz_mag2_hi, double safe) {
    return (unsigned)dz_mag2_hi >= (unsigned)__double2hiint(safe);
}

__device__ __forceinline__ bool not_finite(double v) {
    return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000;
}

// A leap dz <- A dz + B dc.
template <bool CPU>
__device__ __forceinline__ void leap_delta(const double4 e, double& dzx, double& dzy, double dcx, double dcy) {
    double nx, ny;
    if (CPU) {
        nx = (e.x * dzx - e.y * dzy) + (e.z * dcx - e.w * dcy);
        ny = (e.x * dzy + e.y * dzx) + (e.z * dcy + e.w * dcx);
    } else {
        nx = fma(e.x, dzx, fma(-e.y, dzy, fma(e.z, dcx, -e.w * dcy)));
        ny = fma(e.x, dzy, fma(e.y, dzx, fma(e.z, dcy, e.w * dcx)));
    }
    dzx = nx;
    dzy = ny;
}

// One step of the delta at the orbit value (rx, ry), in the profile's roundings.
template <int ARITH, int FT>
__device__ __forceinline__ void delta_step(const ApFrameParams& p, double rx, double ry, double& dzx, double& dzy,
                                           double dcx, double dcy) {
    constexpr bool kCpu = (ARITH == AP_ARITH_REF_CPU);
    constexpr bool kFast = (ARITH == AP_ARITH_FAST);
    if (FT == kFtQuad) {
        double nx, ny;
        if (kFast) {  // (2Z + dz) dz + dc with a = 2Z + dz rounded once
            const double ax = fma(2.0, rx, dzx), ay = fma(2.0, ry, dzy);
            nx = fma(ax, dzx, fma(-ay, dzy, dcx));
            ny = fma(ax, dzy, fma(ay, dzx, dcy));
        } else if (kCpu) {
            nx = twice_plus(rx, dzx) * dzx - twice_plus(ry, dzy) * dzy + dcx;
            ny = twice_plus((rx + dzx) * dzy + ry * dzx, dcy);
        } else {
            nx = fma(twice_plus(rx, dzx), dzx, fma(-twice_plus(ry, dzy), dzy, dcx));
            ny = twice_plus(fma(rx + dzx, dzy, ry * dzx), dcy);
        }
        dzx = nx;
        dzy = ny;
    } else if (FT == kFtShip) {
        const double zx = rx + dzx, zy = ry + dzy;
        if (kFast) {  // 2Z + dz rounded once (2Z is exact); products fused into the sums
            const double ax = fma(2.0, rx, dzx), ay = fma(2.0, ry, dzy);
            const double nx = fma(ax, dzx, fma(-ay, dzy, dcx));
            const double ddx = fold_delta(rx, zx, dzx, ax), ddy = fold_delta(ry, zy, dzy, ay);
            dzy = fma(2.0, fma(fabs(rx), ddy, fma(fabs(ry), ddx, ddx * ddy)), -dcy);
            dzx = nx;
        } else {
            const double ax = twice_plus(rx, dzx), ay = twice_plus(ry, dzy);
            const double nx = ax * dzx - ay * dzy + dcx;
            const double ddx = fold_delta(rx, zx, dzx, ax), ddy = fold_delta(ry, zy, dzy, ay);
            dzy = twice_plus(fabs(rx) * ddy + fabs(ry) * ddx + ddx * ddy, -dcy);
            dzx = nx;
        }
    } else if (kFast) {
        // (Z + dz)^n - Z^n by P_{j+1} = P_j Z + (P_j + Z^j) dz, each complex product
        // sum as one chain of fused multiply-adds, then + k dz + dc
        double pr = dzx, pi = dzy, qr = rx, qi = ry;
        for_powers(p.gen_n, [&]() {
            const double sr = pr + qr, si = pi + qi;
            const double npr = fma(pr, rx, fma(-pi, ry, fma(sr, dzx, -si * dzy)));
            const double npi = fma(pr, ry, fma(pi, rx, fma(sr, dzy, si * dzx)));
            const double nqr = fma(qr, rx, -qi * ry), nqi = fma(qr, ry, qi * rx);
            pr = npr;
            pi = npi;
            qr = nqr;
            qi = nqi;
        });
        const double ox = dzx, oy = dzy;
        dzx = fma(p.gen_kr, ox, fma(-p.gen_ki, oy, pr + dcx));
        dzy = fma(p.gen_kr, oy, fma(p.gen_ki, ox, pi + dcy));
    } else {
        double pr = dzx, pi = dzy, qr = rx, qi = ry;
        for_powers(p.gen_n, [&]() {
            const double t1r = pr * rx - pi * ry, t1i = pr * ry + pi * rx;
            const double sr = pr + qr, si = pi + qi;
            const double t2r = sr * dzx - si * dzy, t2i = sr * dzy + si * dzx;
            pr = t1r + t2r;
            pi = t1i + t2i;
            const double nqr = qr * rx - qi * ry, nqi = qr * ry + qi * rx;
            qr = nqr;
            qi = nqi;
        });
        const double kzr = p.gen_kr * dzx - p.gen_ki * dzy;
        const double kzi = p.gen_kr * dzy + p.gen_ki * dzx;
        dzx = pr + kzr + dcx;
        dzy = pi + kzi + dcy;
    }
}

// Whether the kSpan steps from here on are plain (ap_pack.cu's orbit_window, the low word of the
// record's third slot): |dz|^2's exponent in the record's window, and |dc|^2's at least 60 below it
// (dc_exp60: that exponent plus 60; a |dc|^2 that underflows has exponent 0, and is covered).  Without
// leaps only the window's end counts, and a smaller |dz| stays below what one of 2^30 |dc| grows to
// (960x540 at 1e-26 without leaps, where deltas stay near |dc| for thousands of steps: 12.1 ms
// without spans, 13.6 with spans from 2^30 |dc| on, 6.9 so).
__device__ __forceinline__ int dc_exponent60(double dcx, double dcy) {
    return (int)((unsigned)__double2hiint(dcx * dcx + dcy * dcy) >> 20) + 60;
}
template <bool BLA>
__device__ __forceinline__ bool span_fits(int dz_mag2_hi, const double4 rec, int dc_exp60) {
    const int e = (unsigned)dz_mag2_hi >> 20, w = __double2loint(rec.z);  // unsigned: no NaN fits
    if (!BLA) return max(e, dc_exp60) < (w & 0xffff);
    return e < (w & 0xffff) && e >= dc_exp60 && e >= (__double2hiint(rec.w) >> 20) + (w >> 16);
}

// kSpan steps from record `rec` on without a test: 7 instructions a step where a tested one takes
// about 28.  Lanes that do not fit wait for those that do.  In a pass with leaps the lanes that took a
// span go on into the tested step or the leap of the same loop iteration, together with the others: at
// 1e-26, where lanes fall out of step, 1920x1080 with one-pass rebasing 19.2 ms with a test of the
// next span instead, 17.1 so, 18.3 without spans.  Without leaps nearly all lanes fit again (1e-160:
// 9.7 ms against 10.4).  Taking a span only where most lanes fit measured slower (1e-160: 1.67 ms
// against 1.50), and the Burning Ship, whose lanes disagree more, loses (a 167x167 tile at depth 65541
// 18.8 ms without spans, 28 with): it takes none.
template <int ARITH, int FT>
__device__ __forceinline__ void span_steps(const ApFrameParams& p, const double4* __restrict__ rec, double& dzx,
                                           double& dzy, double dcx, double dcy) {
#pragma unroll
    for (int j = 0; j < kSpan; ++j) {
        const double2 Z = __ldg(reinterpret_cast<const double2*>(rec + j));
        delta_step<ARITH, FT>(p, Z.x, Z.y, dzx, dzy, dcx, dcy);
    }
}

// What a lane does at the end of a loop iteration.  The loops below decide it in the branches of
// their tests and act on it afterwards.  For Multibrot, whose step is 30 to 60 FP64 operations,
// the decision goes through value_barrier, so that all lanes that step do so together: with the
// branches threaded to their ends (a jump from a test to the loop's head) the lanes that passed a
// test and those that skipped it ran the step one after the other, and a step's FP64 instructions
// were issued 1.7 times (a 399x399 tile with n = 4: 8.0 ms, 5.9 with the barrier).  The cheaper
// steps lose more by the barrier than by that (a 1920x1080 Mandelbrot view 1.58 -> 1.78 ms).
enum { kActStep = 0, kActMoved = 1, kActEscaped = 2, kActNotFinite = 3 };
__device__ __forceinline__ void value_barrier(int& v) { asm volatile("" : "+r"(v)); }

// Stage 1.  TAIL: the reference has a periodic tail, whose steps are visited (a 1e-160 frame, whose
// reference has none, with the visits' bound in the loop 1.26 ms, without it 1.24; with one-pass
// rebasing 1.18 and 1.09).  SPANS: z^2 + c whose runs of plain steps are taken as spans.
template <int ARITH, int FT, bool BLA, bool BUDGET, bool TAIL, bool SPANS, class Store>
__device__ __forceinline__ void stage1_advance(const ApFrameParams& p, const ApFrameBuffers& b, PixelRun& s,
                                               Round& round, Store& C, int q) {
    constexpr bool kCpu = (ARITH == AP_ARITH_REF_CPU);
    constexpr bool kMerge = (FT == kFtMulti);
    const bool julia = (p.fractal_type == 2 || p.fractal_type == 3);
    const int ref_len = p.ref_len, max_iter = p.max_iter;
    const double4* __restrict__ orb = reinterpret_cast<const double4*>(b.orbit_packed);
    int k = s.k, glitch = s.glitch, leaps = s.leaps, skipped = s.skipped;
    SampleOut o = s.o;
    double dzx = s.dzx, dzy = s.dzy;
    const double dcpx = julia ? 0.0 : s.dcx, dcpy = julia ? 0.0 : s.dcy;
    const bool strict = p.strict_glitch > 0;
    const bool esc_glitch = (p.flags & AP_FLAG_ESCAPE_GLITCH) != 0;
    const double* __restrict__ R = b.bla_packed;
    const double4* __restrict__ AB =
        reinterpret_cast<const double4*>(b.bla_packed + (size_t)ref_len * 16);
    const int max_level = p.bla_levels - 1;
    bool paused = false;
    int act = kActStep;
    double esc_mag2 = 0.0;
    const int dc_exp60 = dc_exponent60(dcpx, dcpy);
    // the loop runs to `bound`: the orbit's end, or the next visited step of its tail
    // (past step 15, from which on the Pauldelbrot test looks at every step)
    int bound = TAIL ? min(ref_len, max(k, max(16, orbit_tail(orb, ref_len).s0))) : ref_len;
    for (;;) {
        if (k >= bound) {
            if (!TAIL || k >= ref_len) break;
            const OrbitTail tail = orbit_tail(orb, ref_len);
            int gap = tail_gap(C, q, tail, k, false);
            if (gap == 0) {
                const int dk = cycle_visit(C, q, dzx, dzy, k, k);
                if (dk > 0) {
                    const int jump = (ref_len - 1 - k) / dk * dk;
                    k += jump;
                    skipped += jump;
                }
                gap = tail_gap(C, q, tail, k, true);
            }
            bound = gap < ref_len - k ? k + gap : ref_len;
        }
        if (BUDGET && round.over()) {
            paused = true;
            break;
        }
        double4 Z = ldg4(orb + k);
        double dz_mag2 = dzx * dzx + dzy * dzy;
        if (SPANS && k + kSpan <= bound && span_fits<BLA>(__double2hiint(dz_mag2), Z, dc_exp60)) {
            span_steps<ARITH, FT>(p, orb + k, dzx, dzy, dcpx, dcpy);
            k += kSpan;
            if (!BLA || k >= bound) continue;
            Z = ldg4(orb + k);
            dz_mag2 = dzx * dzx + dzy * dzy;
        }
        const double rx = Z.x, ry = Z.y;
        const int dz_hi = __double2hiint(dz_mag2);
        // One branch on the common path: inside the safe radius (no test can fire)
        // and outside the level-0 BLA radius (no leap), the step runs straight
        // through.  The packed radii are 0 wherever k + 2^d >= ref_len, so no level
        // is admissible at the last step without a separate bound check.
        const bool unsafe = outside(dz_hi, Z.z);
        const bool leap = BLA && (dz_mag2 < Z.w);
        act = kActStep;
        if (unsafe || leap) {
            if (unsafe) {
                const double zx = rx + dzx, zy = ry + dzy;
                const double mag2 = zx * zx + zy * zy;
                const double r_mag2 = rx * rx + ry * ry;
                if (mag2 > kBailout) {
                    if (esc_glitch && strict && k > 15 && r_mag2 < 4.0) glitch = 1;
                    esc_mag2 = mag2;
                    act = kActEscaped;
                } else {
                    // the Pauldelbrot threshold, as the reference forms it
                    const double thr = r_mag2 > 1e-8 ? 1e-6 * r_mag2 : -1.0;
                    if (strict && k > 15 && mag2 < thr) glitch = 1;
                }
            }
            if (leap && act == kActStep) {
                int hi = max_level;
                if (dz_mag2 == 0.0 && (dzx != 0.0 || dzy != 0.0)) hi = min(hi, 8);
                const int lo = leap_level(R + (size_t)k * 16, dz_mag2, hi);
                leap_delta<kCpu>(ldg4(AB + (size_t)k * 16 + lo), dzx, dzy, dcpx, dcpy);
                act = kActNotFinite;
                if (!not_finite(dzx) && !not_finite(dzy)) {
                    act = kActMoved;
                    k += 1 << lo;
                    ++leaps;
                    skipped += 1 << lo;
                }
            }
        }
        if (kMerge) value_barrier(act);
        if (act >= kActEscaped) break;
        if (act == kActStep) {
            delta_step<ARITH, FT>(p, rx, ry, dzx, dzy, dcpx, dcpy);
            ++k;
        }
    }
    if (paused) {
        s.dzx = dzx;
        s.dzy = dzy;
        s.k = k;
        s.glitch = glitch;
        s.leaps = leaps;
        s.skipped = skipped;
        return;
    }
    if (act >= kActEscaped) {
        if (act == kActEscaped) {
            o = escaped_sample(k, esc_mag2, inv_ln_for(p.fractal_type, p.gen_n));
        } else {
            o = interior_sample();
            o.s = (float)k;
            o.s64 = (double)k;
            o.k = k;
            glitch = 1;
        }
        s.stage = 3;
    } else {
        // Stage 2: past the end of the reference orbit, iterate z directly.
        const double4 Zend = ldg4(orb + ref_len);
        s.zx = Zend.x + dzx;
        s.zy = Zend.y + dzy;
        if (ref_len < max_iter) glitch = 1;
        s.k2 = k;
        o = interior_sample();
        s.stage = 2;
    }
    s.k = k;
    s.glitch = glitch;
    s.leaps = leaps;
    s.skipped = skipped;
    s.o = o;
}

// Stage 2: direct iteration past the end of the reference.
template <int FT, bool BUDGET, class Store>
__device__ __forceinline__ void stage2_advance(const ApFrameParams& p, PixelRun& s, Round& round, Store& C, int q) {
    const bool julia = (p.fractal_type == 2 || p.fractal_type == 3);
    const int max_iter = p.max_iter;
    const double inv_ln = inv_ln_for(p.fractal_type, p.gen_n);
    int k = s.k, glitch = s.glitch, skipped = s.skipped;
    SampleOut o = s.o;
    double zx = s.zx, zy = s.zy;
    const double cx = julia ? p.julia_cx_hi : p.ref_cx + s.dcx;
    const double cy = julia ? p.julia_cy_hi : p.ref_cy + s.dcy;
    const bool nan_guard = (p.flags & AP_FLAG_NAN_GUARD) != 0;
    bool paused = false;
    constexpr int kKind = FT == kFtQuad ? kKindQuad : FT == kFtShip ? kKindShip : kKindMulti;
    const bool growing = fp64_growing(kKind, cx, cy, p.gen_n, p.gen_kr, p.gen_ki);
    const bool doubles = fp64_doubles(zy, cy);
    CycleStore<1> R;  // in registers: visited after every block
    R.visits[0] = 0;
    int tested = 0;  // steps to test one by one before the next block
    while (k < max_iter) {
        if (BUDGET && round.over()) {
            paused = true;
            break;
        }
        // blocks tested at their end only, as in direct iteration (fp64_orbit, ap_fp64.cuh)
        if (growing && tested == 0 && max_iter - k >= kBlock) {
            const double bx = zx, by = zy;
            for_degree(kKind, p.gen_n, doubles, [&](auto n) {
#pragma unroll
                for (int t = 0; t < kBlock; ++t)
                    fp64_step<AP_ARITH_REF_CUDA, kKind, n()>(zx, zy, zx * zx, zy * zy, cx, cy, p.gen_n, p.gen_kr,
                                                             p.gen_ki);
            });
            if (zx * zx + zy * zy <= kBailout) {
                k += kBlock;
                // a state that repeats never escapes
                if ((BUDGET ? cycle_visit(C, q, zx, zy, k, -1) : cycle_visit(R, 0, zx, zy, k, -1)) > 0) {
                    s.k2 += max_iter - k;
                    skipped += max_iter - k;
                    k = max_iter;
                }
                continue;
            }
            zx = bx;
            zy = by;
            tested = kBlock + 1;
        }
        if (tested > 0) --tested;
        const double zx2 = zx * zx, zy2 = zy * zy;
        const double mag2 = zx2 + zy2;
        if (nan_guard && (isnan(mag2) || isinf(mag2))) {
            o.s = (float)k;
            o.s64 = (double)k;
            o.k = k;
            glitch = 1;
            break;
        }
        if (mag2 > kBailout) {
            o = escaped_sample(k, mag2, inv_ln);
            break;
        }
        if (FT == kFtQuad) {
            zy = 2.0 * zx * zy + cy;
            zx = zx2 - zy2 + cx;
        } else if (FT == kFtShip) {
            zy = 2.0 * fabs(zx) * fabs(zy) - cy;
            zx = zx2 - zy2 + cx;
        } else {
            double zr = zx, zi = zy;
            for_powers(p.gen_n, [&]() {
                const double nr = zr * zx - zi * zy, ni = zr * zy + zi * zx;
                zr = nr;
                zi = ni;
            });
            const double kzr = p.gen_kr * zx - p.gen_ki * zy;
            const double kzi = p.gen_kr * zy + p.gen_ki * zx;
            zx = zr + kzr + cx;
            zy = zi + kzi + cy;
        }
        ++k;
    }
    s.zx = zx;
    s.zy = zy;
    if (!paused) s.stage = 3;
    s.k = k;
    s.glitch = glitch;
    s.skipped = skipped;
    s.o = o;
}

// Both stages of a single-reference pixel.  The lanes of a warp enter stage 2 together: the barrier
// keeps the compiler from going from a loop's exit straight into it, lane by lane (a 437x437 view at
// 5e-27 with a short reference 2.07 ms, 1.47 with it).
template <int ARITH, int FT, bool BLA, bool BUDGET, bool SPANS, class Store>
__device__ __forceinline__ void pixel_advance(const ApFrameParams& p, const ApFrameBuffers& b, PixelRun& s,
                                              Round round, bool tail, Store& C, int q) {
    if (s.stage == 1) {
        if (tail) stage1_advance<ARITH, FT, BLA, BUDGET, true, SPANS>(p, b, s, round, C, q);
        else stage1_advance<ARITH, FT, BLA, BUDGET, false, SPANS>(p, b, s, round, C, q);
    }
    value_barrier(s.stage);
    if (s.stage == 2) stage2_advance<FT, BUDGET>(p, s, round, C, q);
}

// One-pass rebasing (AP_FLAG_REBASE), for orbits that start at Z_0 = 0 (fractal
// types 0, 1, 4).  k counts the pixel's iterations, m indexes the reference.  At
// each step z = Z_m + dz is tested for escape; when |z| < |dz| -- the delta has
// outgrown the value it perturbs, where a plain delta would lose its precision --
// or when the reference has ended (m == ref_len), the delta restarts from the start
// of the orbit: dz <- z, m <- 0 (Zhuoran, fractalforums.org 2021).  A pixel is never
// flagged glitched (only a NaN/Inf delta is) and never falls back to direct
// iteration, so one pass serves every pixel.  The packed safe radius also rules
// out the rebase test (|dz| < |Z|/2), so the common path is the same single branch
// as pixel_advance's.  Leaps are capped so that k never passes max_iter.  ARITH may
// also be AP_ARITH_FAST: |dz|^2, |z|^2 and every formula's step as fused multiply-adds
// (about 10 FP64 instructions per Mandelbrot step on the common path; a Multibrot
// power costs 14 instead of 22), leaps as the CUDA profile.
template <int ARITH, int FT, bool BLA, bool BUDGET, bool TAIL, bool SPANS, class Store>
__device__ __forceinline__ void rebase_advance(const ApFrameParams& p, const ApFrameBuffers& b, PixelRun& s,
                                               Round round, Store& C, int q) {
    constexpr bool kCpu = (ARITH == AP_ARITH_REF_CPU);
    constexpr bool kFast = (ARITH == AP_ARITH_FAST);
    constexpr bool kMerge = (FT == kFtMulti);
    const int ref_len = p.ref_len, max_iter = p.max_iter;
    const double4* __restrict__ orb = reinterpret_cast<const double4*>(b.orbit_packed);
    const double* __restrict__ R = b.bla_packed;
    const double4* __restrict__ AB = reinterpret_cast<const double4*>(b.bla_packed + (size_t)ref_len * 16);
    const int max_level = p.bla_levels - 1;
    const double dcpx = s.dcx, dcpy = s.dcy;
    // k (the pixel's iterations) is not kept: a step or a leap moves k and m alike and a
    // restart moves only m, so k = m + (max_iter - lim) with lim moved at each restart,
    // and the loop runs while m < lim (k < max_iter).
    int m = s.m, lim = max_iter - s.k + s.m;
    int leaps = s.leaps, skipped = s.skipped, rebases = s.rebases;
    double dzx = s.dzx, dzy = s.dzy;
    bool paused = false;
    int act = kActStep;
    double esc_mag2 = 0.0;
    const int dc_exp60 = dc_exponent60(dcpx, dcpy);
    // A restart at an orbit that starts at 0, without a leap there, needs no test at m = 0: z = dz has
    // just been tested.  Multibrot goes straight to the step (a 504x504 view of bounded pixels 11.2 ->
    // 8.0 ms); Mandelbrot frames lose by it (1920x1080 at 1e-160 1.19 ms, 1.24 with it), and so does the
    // Burning Ship (800x451 at depth 65541 25.9 and 29.0).
    constexpr bool kStepOn = FT == kFtMulti;
    // the Burning Ship restarts often and settles on a cycle rarely (127x127 at depth 12433: a visit at
    // every restart 4.8 ms, every eighth 3.8, every 16th 3.6)
    constexpr int kRestartStride = FT == kFtShip ? 32 : 4;
    const double4 Zstart = kStepOn ? ldg4(orb) : make_double4(1.0, 0.0, 0.0, 0.0);
    const bool step_on = kStepOn && Zstart.x == 0.0 && Zstart.y == 0.0 && !(Zstart.w > 0.0);
    // the loop runs to `bound`: lim, or the next visited step of the reference's tail
    const int tail_s0 = TAIL ? max(1, orbit_tail(orb, ref_len).s0) : INT_MAX;
    int bound = min(lim, max(m, tail_s0));
    for (;;) {
        if (!TAIL) bound = lim;
        if (m >= bound) {
            if (!TAIL || m >= lim) break;
            const OrbitTail tail = orbit_tail(orb, ref_len);
            int gap = tail_gap(C, q, tail, m, false);
            if (gap == 0) {
                const int k = m + (max_iter - lim);
                const int dk = cycle_visit(C, q, dzx, dzy, k, m);
                if (dk > 0) {
                    // no restart in the cycle: it moves m too and has to end below the orbit's end
                    // (it closed at an earlier step); else m returns with it
                    const bool moves = C.m[q] != m;
                    const int room = moves ? min(lim - m, ref_len - 1 - m) : lim - m;
                    const int jump = max(0, room) / dk * dk;
                    if (moves) m += jump;
                    else lim -= jump;
                    skipped += jump;
                }
                gap = tail_gap(C, q, tail, m, true);
            }
            bound = gap < lim - m ? m + gap : lim;
            if (m >= lim) break;
        }
        if (BUDGET && round.over()) {
            paused = true;
            break;
        }
        double4 Z = ldg4(orb + m);
        double dz_mag2 = kFast ? fma(dzx, dzx, dzy * dzy) : dzx * dzx + dzy * dzy;
        if (SPANS && m + kSpan <= bound && span_fits<BLA>(__double2hiint(dz_mag2), Z, dc_exp60)) {
            span_steps<ARITH, FT>(p, orb + m, dzx, dzy, dcpx, dcpy);
            m += kSpan;
            if (!BLA || m >= bound) continue;
            Z = ldg4(orb + m);
            dz_mag2 = kFast ? fma(dzx, dzx, dzy * dzy) : dzx * dzx + dzy * dzy;
        }
        double rx = Z.x, ry = Z.y;
        const int dz_hi = __double2hiint(dz_mag2);
        // ap_pack_orbit leaves the orbit's last record (m == ref_len) with safe radius 0,
        // so the end of the reference takes this branch without a test of its own
        const bool unsafe = outside(dz_hi, Z.z);
        const bool leap = BLA && (dz_mag2 < Z.w);
        act = kActStep;
        if (unsafe || leap) {
            bool may_leap = leap;
            if (unsafe) {
                const double zx = rx + dzx, zy = ry + dzy;
                const double mag2 = kFast ? fma(zx, zx, zy * zy) : zx * zx + zy * zy;
                if (!(mag2 <= kBailout)) {
                    esc_mag2 = mag2;
                    act = kActEscaped;
                } else if (mag2 < dz_mag2 || (m == ref_len && m > 0)) {
                    dzx = zx;
                    dzy = zy;
                    lim -= m;
                    m = 0;
                    ++rebases;
                    const int dk = rebases > kFirstRestart && rebases % kRestartStride == 0 ? cycle_visit(C, q, dzx, dzy, max_iter - lim, 0) : 0;
                    if (dk > 0) {
                        const int jump = lim / dk * dk;
                        lim -= jump;
                        skipped += jump;
                    }
                    bound = min(lim, tail_s0);
                    act = step_on && lim > 0 ? kActStep : kActMoved;
                    if (kStepOn) {
                        rx = 0.0;
                        ry = 0.0;
                        may_leap = false;
                    }
                }
            }
            if (may_leap && act == kActStep) {
                int hi = max_level;
                if (dz_mag2 == 0.0 && (dzx != 0.0 || dzy != 0.0)) hi = min(hi, 8);
                hi = min(hi, 31 - __clz(lim - m));  // k + 2^lo <= max_iter
                const int lo = leap_level(R + (size_t)m * 16, dz_mag2, hi);
                leap_delta<kCpu>(ldg4(AB + (size_t)m * 16 + lo), dzx, dzy, dcpx, dcpy);
                act = kActNotFinite;
                if (!not_finite(dzx) && !not_finite(dzy)) {
                    act = kActMoved;
                    m += 1 << lo;
                    ++leaps;
                    skipped += 1 << lo;
                }
            }
        }
        if (kMerge) value_barrier(act);
        if (act >= kActEscaped) break;
        if (act == kActStep) {
            delta_step<ARITH, FT>(p, rx, ry, dzx, dzy, dcpx, dcpy);
            ++m;
        }
    }
    const int k = m + (max_iter - lim);
    if (!paused) {
        s.stage = 3;
        if (act == kActEscaped && !isnan(esc_mag2)) {
            s.o = escaped_sample(k, esc_mag2, inv_ln_for(p.fractal_type, p.gen_n));
        } else if (act >= kActEscaped) {
            s.o = interior_sample();
            s.o.s = (float)k;
            s.o.s64 = (double)k;
            s.o.k = k;
            s.glitch = 1;
        }
    }
    s.dzx = dzx;
    s.dzy = dzy;
    s.k = k;
    s.m = m;
    s.leaps = leaps;
    s.skipped = skipped;
    s.rebases = rebases;
}

__device__ __forceinline__ void pixel_finish(const ApFrameParams& p, const ApFrameBuffers& b, const PixelRun& s) {
    const int max_iter = p.max_iter;
    const int k_end = (s.o.k == -1) ? max_iter : s.k;
    b.iter_map[s.idx] = s.o.s;
    if (b.kmap) b.kmap[s.idx] = s.o.k;
    if (b.s64) b.s64[s.idx] = s.o.s64;
    if (b.glitch_out) b.glitch_out[s.idx] = s.glitch ? 1 : 0;
    if (b.counters) {
        const int it1 = (s.k2 < 0 ? k_end - s.k0 : s.k2 - s.k0) - s.skipped;
        const int it2 = s.k2 < 0 ? 0 : k_end - s.k2;
        reinterpret_cast<int4*>(b.counters)[s.idx] = make_int4(it1, s.leaps, it2, s.rebases);
    }
}

// One pixel (i, j) of a coarse pass, start to finish (REBASE: AP_FLAG_REBASE).  The tail is the orbit's,
// so all pixels of a pass take one of the two loops.
template <int ARITH, int FT, bool BLA, bool REBASE, bool SPANS>
__device__ __forceinline__ void coarse_pixel(const ApFrameParams& p, const ApFrameBuffers& b, int i,
                                             int j) {
    PixelRun s;
    if (!pixel_begin<ARITH, FT>(p, b, i, j, s)) return;
    CycleLocal C;
    C.visits[0] = 0;
    // one reference's Multibrot and Burning Ship loops run no faster without the visits
    const bool tail = (!REBASE && FT != kFtQuad) || has_tail(reinterpret_cast<const double4*>(b.orbit_packed), p.ref_len);
    if (REBASE) {
        if (tail) rebase_advance<ARITH, FT, BLA, false, true, SPANS>(p, b, s, Round{}, C, 0);
        else rebase_advance<ARITH, FT, BLA, false, false, SPANS>(p, b, s, Round{}, C, 0);
    } else {
        pixel_advance<ARITH, FT, BLA, false, SPANS>(p, b, s, Round{}, tail, C, 0);
    }
    pixel_finish(p, b, s);
}

}  // namespace ap
