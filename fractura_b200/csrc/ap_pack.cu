// ap_pack.cu -- device re-layout of the reference orbit and the BLA table into
// the records the perturbation kernels read (one load per step, one 128-byte
// row per level search).  Values are copied or computed exactly as the
// per-step code computes them, so results do not change.
#include "ap_common.cuh"

namespace ap {

// The radius below which no test of a step at |Z| = rz can fire (see pack_orbit_kernel).
__device__ __forceinline__ double safe_radius(double rz) {
    const double s = fmin(256.0 * (1.0 - 1e-12) - rz * (1.0 + 1e-12), rz * (1.0 - 1e-12) * 0.5 * (1.0 - 1e-7));
    return s > 0.0 ? s : 0.0;
}

// The window of |dz| at step k in which the next kSpan steps of z^2 + c are plain: no test of
// theirs can fire and none of them leaps.  While |dz_j| is below step j's
// safe radius it is at most |Z_j| / 2, so
//     1.5 |Z_j| |dz_j| - |dc|  <=  |dz_{j+1}|  <=  2.5 |Z_j| |dz_j| + |dc|
// (|dz'| = |2 Z + dz| |dz| up to dc).  With the factors widened to 1.49 and 2.51, which cover
// every rounding and a |dc| up to 2^-29 |dz_0| (the kernels check that) as long as the lower
// products stay above 2^-20, the window is |dz_0| < h = min_j s_j / prod_{i<j} 2.51 |Z_i| and,
// with leaps, |dz_0| >= max_j r_j / prod_{i<j} 1.49 |Z_i|.  The level-0 radii r_j of ap_build_bla
// and ap_build_bla_dc are proportional to |Z_j|, so that bound is r_k times a number of the orbit
// alone.  Kept: h^2's biased exponent (0: no window) and, above it, two more than the exponent of
// that number squared, which the kernels add to r_k^2's.
__device__ __forceinline__ unsigned orbit_window(const double* __restrict__ re, const double* __restrict__ im, int k,
                                                 int n) {
    if (k == 0 || k + kSpan >= n) return 0u;  // step 0 may have radius 0 next to 0
    double up = 1.0, down = 1.0, h = 256.0, l = 0.0, rk = 0.0;
    for (int j = 0; j < kSpan; ++j) {
        const double rz = sqrt(re[k + j] * re[k + j] + im[k + j] * im[k + j]);
        if (j == 0) rk = rz;
        if (!(down >= 0x1p-20) || !(rk > 0.0)) return 0u;
        h = fmin(h, safe_radius(rz) / (up * (1.0 + 1e-9)));
        l = fmax(l, rz / rk * (1.0 + 1e-9) / down);
        up *= 2.51 * rz;
        down *= 1.49 * rz;
    }
    const unsigned end = (unsigned)__double2hiint(h * h) >> 20;
    const unsigned first = ((unsigned)__double2hiint(l * l) >> 20) - 1023u + 2u;  // l >= 1
    return end > 0u && first < 0x8000u ? (first << 16) | end : 0u;
}

// The periodic tail of an orbit of n values, for the kernels' cycle detection: the smallest
// period p <= 4095 with Z_k = Z_{k-p} (bit for bit up to the sign of a zero) for the orbit's last 8 steps,
// and the s0 from which on it holds for every k from s0 + p to n - 2; kept as -(4096 s0 + p) in the last
// record (orbit_tail, ap_coarse.cuh, asks for two periods and 64 steps of it), 0 when there is none.  An
// orbit that escaped has none (its last value tells).  One block of a launch of `blocks`: it searches the
// period for itself, all candidates' first values at once, compares its share of the orbit and returns
// the word of that (the largest s0 of all shares is the largest word), the same in all its threads.
constexpr int kTailThreads = 256, kTailMaxPeriod = 4095;
__device__ double tail_word(const double* __restrict__ re, const double* __restrict__ im, int n, int block, int blocks) {
    __shared__ int period_s, bad_s;
    const int last = n - 2;  // the record at n - 1 is the orbit's end, never a step
    if (last < 128 || !(re[n - 1] * re[n - 1] + im[n - 1] * im[n - 1] <= kBailout)) return 0.0;
    const int t = threadIdx.x;
    if (t == 0) {
        period_s = kTailMaxPeriod + 1;
        bad_s = -1;
    }
    __syncthreads();
    constexpr int kEach = (kTailMaxPeriod + 1) / kTailThreads;
    const double lx = re[last], ly = im[last];
    unsigned maybe = 0u;
#pragma unroll
    for (int i = 0; i < kEach; ++i) {
        const int p = 1 + t + kTailThreads * i;
        if (p <= kTailMaxPeriod && 2 * p < last && lx == re[last - p] && ly == im[last - p]) maybe |= 1u << i;
    }
    for (; maybe != 0u; maybe &= maybe - 1u) {
        const int p = t + kTailThreads * (__ffs(maybe) - 1) + 1;
        bool same = true;
        for (int j = 1; j < 8 && same; ++j) same = re[last - j] == re[last - j - p] && im[last - j] == im[last - j - p];
        if (same) {
            atomicMin(&period_s, p);
            break;
        }
    }
    __syncthreads();
    const int p = period_s;
    if (p > kTailMaxPeriod) return 0.0;
    int bad = -1;  // the largest k of this block's share with Z_k != Z_{k-p}
#pragma unroll 4
    for (long long k = (long long)p + block * kTailThreads + t; k <= last; k += blocks * kTailThreads)
        if (!(re[k] == re[k - p] && im[k] == im[k - p])) bad = (int)k;
    if (bad >= 0) atomicMax(&bad_s, bad);
    __syncthreads();
    const int s0 = bad_s < 0 ? 0 : bad_s + 1 - p;
    return -(4096.0 * (double)s0 + (double)p);
}

// Long orbits (from kLongOrbit values): shared out over the blocks of a kernel of its own.  On one block of
// the packing kernel 200000 values held every frame of a bounded reference up for 306 us (23 so), 16000
// for 19 (19 so); a short orbit would pay for the second launch (6000 values without a tail 9 us, 12.5
// with it; 8050 of an escaped one 6.4 and 8).
constexpr int kLongOrbit = 1 << 14;
__global__ void __launch_bounds__(kTailThreads) pack_tail_kernel(const double* __restrict__ re,
                                                                 const double* __restrict__ im, int n,
                                                                 double4* __restrict__ out) {
    const double word = tail_word(re, im, n, blockIdx.x, gridDim.x);
    if (threadIdx.x == 0 && word < 0.0)  // negative: the bits order by magnitude
        atomicMax(reinterpret_cast<unsigned long long*>(&out[n - 1].w), (unsigned long long)__double_as_longlong(word));
}

__global__ void __launch_bounds__(256) pack_orbit_kernel(const double* __restrict__ re,
                                                         const double* __restrict__ im, int n,
                                                         double4* __restrict__ out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    // a short orbit's tail: the last block, which writes the last record
    const double tail = n < kLongOrbit && blockIdx.x == gridDim.x - 1 ? tail_word(re, im, n, 0, 1) : 0.0;
    if (k >= n) return;
    const double rx = re[k], ry = im[k];
    const double r_mag2 = rx * rx + ry * ry;
    // Safe radius s: for |dz| < s the rounded |Z + dz|^2 is neither above the
    // bailout 65536 (|Z| + s <= 256 (1 - 1e-12)), nor below the Pauldelbrot
    // threshold 1e-6 |Z|^2, nor below the rounded |dz|^2 (the rebase test):
    // s <= |Z| (1 - 1e-7) / 2 keeps |Z + dz| >= |Z| - s > s (1 + 1e-7) > |dz|,
    // and 1e-6 |Z|^2 < s^2 covers the Pauldelbrot threshold.  The 1e-12 margins
    // cover the roundings of |Z|, of Z + dz and of the squares.  Stored as
    // s^2 (1 - 1e-12) to be compared with the rounded |dz|^2.
    // The kernels compare high words (one unit down: a delta just below the radius takes the tests
    // too); the low word holds the record's span window.
    double s = safe_radius(sqrt(r_mag2));
    if (k == n - 1) s = 0.0;  // the orbit's end is never a safe step (the rebase kernels rely on it)
    const int safe_hi = __double2hiint(s * s * (1.0 - 1e-12)) - 1;
    const double safe = safe_hi > 0 ? __hiloint2double(safe_hi, (int)orbit_window(re, im, k, n)) : 0.0;
    // slot 3: the level-0 BLA radius, written by ap_pack_bla (0: no leap); in the last record,
    // which no leap starts from, the periodic tail (a long orbit's: by pack_tail_kernel)
    out[k] = make_double4(rx, ry, safe, k == n - 1 ? tail : 0.0);
}

__global__ void __launch_bounds__(256) pack_bla_kernel(const double* __restrict__ T, int levels,
                                                       int ref_len, double* __restrict__ R,
                                                       double4* __restrict__ AB,
                                                       double* __restrict__ orb) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;  // one (k, d) pair per thread
    if (t >= ref_len * 16) return;
    const int k = t >> 4, d = t & 15;
    if (d < levels) {
        const double* e = T + ((size_t)d * ref_len + k) * 5;
        // a level is admissible only if its leap ends before the orbit does
        // (k + 2^d < ref_len); the coarse loop relies on 0 radii elsewhere
        R[t] = (k + (1 << d) < ref_len) ? e[4] : 0.0;
        if (d == 0 && orb) orb[4 * (size_t)k + 3] = R[t];  // the orbit record's level-0 radius
        AB[t] = make_double4(e[0], e[1], e[2], e[3]);
    } else {
        R[t] = 0.0;
        AB[t] = make_double4(0.0, 0.0, 0.0, 0.0);
    }
}

}  // namespace ap

extern "C" int ap_pack_orbit(const double* ref_re, const double* ref_im, int32_t ref_len,
                             double* out, void* stream) {
    if (!ref_re || !ref_im || !out || ref_len < 0 || (reinterpret_cast<uintptr_t>(out) & 31u)) {
        ap::set_error("ap_pack_orbit: bad arguments (out must be 32-byte aligned)");
        return AP_E_INVALID;
    }
    const int n = ref_len + 1;
    ap::pack_orbit_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        ref_re, ref_im, n, reinterpret_cast<double4*>(out));
    const int rc = ap::check_launch("pack_orbit_kernel");
    if (rc != AP_OK || n < ap::kLongOrbit) return rc;
    const int blocks = (n + 2047) / 2048 < 148 ? (n + 2047) / 2048 : 148;
    ap::pack_tail_kernel<<<blocks, ap::kTailThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        ref_re, ref_im, n, reinterpret_cast<double4*>(out));
    return ap::check_launch("pack_tail_kernel");
}

extern "C" int ap_pack_bla(const double* table, int32_t levels, int32_t ref_len, double* out,
                           double* orbit_packed, void* stream) {
    if (!table || !out || levels < 1 || levels > 16 || ref_len < 1 ||
        (reinterpret_cast<uintptr_t>(out) & 31u)) {
        ap::set_error("ap_pack_bla: bad arguments (1 <= levels <= 16, out 32-byte aligned)");
        return AP_E_INVALID;
    }
    double* R = out;
    double4* AB = reinterpret_cast<double4*>(out + (size_t)ref_len * 16);
    const int n = ref_len * 16;
    ap::pack_bla_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        table, levels, ref_len, R, AB, orbit_packed);
    return ap::check_launch("pack_bla_kernel");
}
