// ap_render.cu -- unified render passes (coarse / full supersample / edge
// supersample) for every precision tier, behind ap_render_pass and
// ap_resolve_hist_pass.
//
// Coarse passes run one thread per output pixel; supersampling passes deal the samples of the
// selected pixels to a warp's lanes.
#include <cstdio>

#include "ap_common.cuh"
#include "ap_fp64.cuh"
#include "ap_samples.cuh"
#include "ap_tiers.cuh"

namespace ap {

// Blocks of kTile x kTile pixels (warps of 8 x 4).  A block lives as long as its slowest
// pixel; small blocks let an SM refill as each one ends, instead of holding 8 warps for the
// one long-lived pixel of a 16 x 16 tile.
constexpr int kTile = 8;

template <int TIER, int ARITH, int KIND>
__device__ __forceinline__ SampleOut sample_at(const ApFrameParams& p, const ApFrameBuffers& b,
                                               double sub_i, double sub_j) {
    if constexpr (TIER == AP_TIER_FP64) {
        double x, y;
        if (p.flags & AP_FLAG_MAP_FUSED) {
            x = fma(sub_i, p.dx_hi, p.x_min_hi);
            y = fma(-sub_j, p.dy_hi, p.y_max_hi);
        } else {
            x = p.x_min_hi + sub_i * p.dx_hi;
            y = p.y_max_hi - sub_j * p.dy_hi;
        }
        return fp64_sample<ARITH>(x, y, p);
    } else if constexpr (TIER == AP_TIER_DD) {
        return dd_sample_at<ARITH, KIND == 4>(p, sub_i, sub_j);
    } else if constexpr (TIER == AP_TIER_PERTURB) {
        return perturb_sample_at<ARITH>(p, b, sub_i, sub_j);
    } else {
        return floatexp_sample_at<ARITH, KIND>(p, b, sub_i, sub_j);
    }
}

// One centred sample per pixel (AP_MODE_COARSE): mandelbrot_unified_*_kernel
// (math_core/cuda_kernels.py:1615-1917) outside its supersampling branches.
template <int TIER, int ARITH, int KIND>
__global__ void __launch_bounds__(kTile * kTile) render_pass_kernel(const ApFrameParams p,
                                                          const ApFrameBuffers b) {
    __shared__ Palette palette;
    const bool rgb = !(p.flags & AP_FLAG_NO_RGB), hist_colour = (p.flags & AP_FLAG_HIST_COLOUR) != 0;
    if (rgb) {
        if (threadIdx.x == 0) palette = palette_of(p, hist_colour);
        __syncthreads();
    }
    const int i = blockIdx.x * kTile + (threadIdx.x & (kTile - 1));
    const int j = blockIdx.y * kTile + (threadIdx.x / kTile);
    if (i >= p.width || j >= p.height) return;
    const size_t idx = (size_t)j * p.width + i;
    if (p.rebase_pass > 0 && b.glitch_in[idx] == 0) return;
    constexpr bool kPert = (TIER >= AP_TIER_PERTURB);
    const int f = p.factor;
    const double sub_offset = ((double)f - 1.0) * 0.5;
    const SampleOut o = sample_at<TIER, ARITH, KIND>(p, b, (double)(i * f) + sub_offset,
                                                      (double)(j * f) + sub_offset);
    b.iter_map[idx] = o.s;
    if (b.kmap) b.kmap[idx] = o.k;
    if (b.s64) b.s64[idx] = o.s64;
    if (b.counters) {
        reinterpret_cast<int4*>(b.counters)[idx] = make_int4(o.iters, o.leaps, o.iters2, 0);
    }
    if (kPert && b.glitch_out) b.glitch_out[idx] = o.glitch > 0 ? 1 : 0;
    if (rgb) {
        double r = 0.0, g = 0.0, bb = 0.0;
        if ((double)o.s >= 0.0) colour_of(p, palette, b.lut, b.cdf, hist_colour, (double)o.s, r, g, bb);
        store_rgb(b.rgb, p.is_hdr, idx, r, g, bb);
    }
}

// f x f samples of the selected pixels.
// hist_resolve = 0: the supersampling branches of mandelbrot_unified_*_kernel
//   (math_core/cuda_kernels.py:1615-1917);
// hist_resolve = 1: ssaa_resolve_hist_*_kernel (math_core/cuda_kernels.py:2038-2234).
// Few pixels are selected (edges, glitches), and the lanes of a warp that ran a pixel each would
// be mostly idle and take their f x f samples one after the other.  A warp lists the selected
// pixels of an 8 x 4 patch, takes `share` of them (the share-th of the patch that its block index
// names; most blocks find none and end) and deals out single samples to its lanes; the lane that
// owns a pixel then adds the pixel's colours up in sample order (sy, then sx), so the sums round as
// the sequential loop's.  Measured against a pixel per lane: 1280x720 double-double Burning Ship
// with 2x SSAA 56.6 -> 53.1 ms with one warp a patch.  Its time was then the tail of the patches whose
// pixels are all selected and bounded (four rounds of 20000 steps one after the other); with the
// rounds on warps of their own 53.7 -> 44.1 ms, and a 1283x721 Julia frame 681 -> 645 us.  A pass that
// selects next to nothing pays for the blocks that find none (1280x720, 25 -> 75 us).
template <int TIER, int ARITH, int KIND>
__global__ void __launch_bounds__(32) supersample_kernel(const ApFrameParams p, const ApFrameBuffers b,
                                                         const int hist_resolve, const int share, const int shares) {
    constexpr bool kPert = (TIER >= AP_TIER_PERTURB);
    __shared__ double red[32], green[32], blue[32];
    __shared__ int work[32][4];  // iterations, leaps, stage-2 steps, glitch
    __shared__ uint8_t list[32];
    __shared__ Palette palette;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x;
    const int i0 = (blockIdx.x / shares) * 8, j0 = (blockIdx.z * gridDim.y + blockIdx.y) * 4;
    const int first = (blockIdx.x % shares) * share;
    int i = i0 + (lane & 7), j = j0 + (lane >> 3);
    bool take = i < p.width && j < p.height;
    if (take) {
        const size_t idx = (size_t)j * p.width + i;
        if (p.rebase_pass > 0 && b.glitch_in[idx] == 0) take = false;
        else if (hist_resolve ? p.rebase_pass == 0 : p.mode == AP_MODE_EDGE) take = b.edge_mask[idx] != 0;
    }
    const unsigned sel = __ballot_sync(full, take);
    const int count = min(share, __popc(sel) - first);  // pixels, owned by lanes 0, 1, ...
    if (count <= 0) return;
    const int place = __popc(sel & ((1u << lane) - 1u)) - first;
    if (take && place >= 0 && place < count) list[place] = (uint8_t)lane;
    const bool hist_colour = hist_resolve || (p.flags & AP_FLAG_HIST_COLOUR);
    if (lane == 0) palette = palette_of(p, hist_colour);
    __syncwarp();
    const bool write_iter = hist_resolve ? (p.rebase_pass > 0) : ((p.flags & AP_FLAG_ITER_LAST_SUB) != 0);
    const int f = p.factor, rows = count * f;
    double ra = 0.0, ga = 0.0, ba = 0.0;
    int glitches = 0, iters = 0, leaps = 0, iters2 = 0;
    for (int row0 = 0; row0 < rows; row0 += sample_rows(f)) {
        const int part = min(sample_rows(f), rows - row0), total = part * f;
        // the owned pixel's samples of this part
        const int lo = min(max(lane * f - row0, 0), part) * f, hi = min(max(lane * f + f - row0, 0), part) * f;
        for (int base = 0; base < total; base += 32) {
            const int q = base + lane;
            if (q < total) {
                int pixel, sx, sy;
                sample_place(row0, q, f, &pixel, &sx, &sy);
                const int at = list[pixel];
                i = i0 + (at & 7);
                j = j0 + (at >> 3);
                const SampleOut o = sample_at<TIER, ARITH, KIND>(p, b, (double)(i * f + sx), (double)(j * f + sy));
                double r = 0.0, g = 0.0, bb = 0.0;
                if ((double)o.s >= 0.0) colour_of(p, palette, b.lut, b.cdf, hist_colour, (double)o.s, r, g, bb);
                red[lane] = r;
                green[lane] = g;
                blue[lane] = bb;
                work[lane][0] = o.iters;
                work[lane][1] = o.leaps;
                work[lane][2] = o.iters2;
                work[lane][3] = o.glitch;
                if (write_iter && sx == f - 1 && sy == f - 1) {
                    const size_t idx = (size_t)j * p.width + i;
                    b.iter_map[idx] = o.s;
                    if (b.kmap) b.kmap[idx] = o.k;
                    if (b.s64) b.s64[idx] = o.s64;
                }
            }
            __syncwarp();
            if (lane < count) {
                for (int t = max(lo, base); t < min(hi, base + 32); ++t) {
                    ra += red[t - base];
                    ga += green[t - base];
                    ba += blue[t - base];
                    iters += work[t - base][0];
                    leaps += work[t - base][1];
                    iters2 += work[t - base][2];
                    glitches += work[t - base][3] > 0 ? 1 : 0;
                }
            }
            __syncwarp();
        }
    }
    if (lane < count) {
        i = i0 + (list[lane] & 7);
        j = j0 + (list[lane] >> 3);
        const size_t idx = (size_t)j * p.width + i;
        const double inv = 1.0 / ((double)f * f);
        store_rgb(b.rgb, p.is_hdr, idx, ra * inv, ga * inv, ba * inv);
        if (kPert && b.glitch_out) b.glitch_out[idx] = glitches > 0 ? 1 : 0;
        if (b.counters) reinterpret_cast<int4*>(b.counters)[idx] = make_int4(iters, leaps, iters2, 0);
    }
}

// The pixels a warp takes of its patch: the fewest (from four on, so that a patch is eight blocks at
// most) whose f x f samples leave no more than a sixteenth of the lanes idle in the last round; the
// whole patch for one sample a pixel, and where the marks that choose pixels are the map that the
// pass writes its glitches to, which its other warps may still have to read.
static int patch_share(const ApFrameParams& p, const ApFrameBuffers& b) {
    if (p.factor == 1 || (b.glitch_out && (b.glitch_out == b.glitch_in || b.glitch_out == b.edge_mask))) return 32;
    const long long f2 = (long long)p.factor * p.factor;
    int share = 4;
    while (share < 32 && 16 * share * f2 < 15 * ((share * f2 + 31) / 32 * 32)) ++share;
    return share;
}

template <int TIER, int ARITH, int KIND>
static int launch_pass(const ApFrameParams& p, const ApFrameBuffers& b, int hist_resolve, cudaStream_t st) {
    if (!hist_resolve && p.mode == AP_MODE_COARSE) {
        dim3 grid((p.width + kTile - 1) / kTile, (p.height + kTile - 1) / kTile);
        render_pass_kernel<TIER, ARITH, KIND><<<grid, kTile * kTile, 0, st>>>(p, b);
        return check_launch("render_pass_kernel");
    }
    const int share = patch_share(p, b), shares = (32 + share - 1) / share;
    const int rows = (p.height + 3) / 4, fold = min(rows, 32768);  // a grid's y ends at 65535
    dim3 grid((p.width + 7) / 8 * shares, fold, (rows + fold - 1) / fold);
    supersample_kernel<TIER, ARITH, KIND><<<grid, 32, 0, st>>>(p, b, hist_resolve, share, shares);
    return check_launch("supersample_kernel");
}

// KIND: the formula class (0 z^2 + c, 1 Burning Ship, 4 Multibrot) for the tiers whose samples are
// built for one (double-double separates Multibrot, whose power loop wants more registers, from
// the others); 0 for the tiers that tell formulas apart at run time.
template <int TIER, int ARITH>
static int launch_formula(const ApFrameParams& p, const ApFrameBuffers& b, int hist_resolve, cudaStream_t st) {
    if constexpr (TIER == AP_TIER_DD || TIER == AP_TIER_FLOATEXP) {
        if (p.fractal_type == 4) return launch_pass<TIER, ARITH, 4>(p, b, hist_resolve, st);
    }
    if constexpr (TIER == AP_TIER_FLOATEXP) {
        if (p.fractal_type & 1) return launch_pass<TIER, ARITH, 1>(p, b, hist_resolve, st);
    }
    return launch_pass<TIER, ARITH, 0>(p, b, hist_resolve, st);
}

template <int TIER>
static int launch_arith(const ApFrameParams& p, const ApFrameBuffers& b, int hist_resolve,
                        cudaStream_t st) {
    if (p.arith == AP_ARITH_REF_CPU) return launch_formula<TIER, AP_ARITH_REF_CPU>(p, b, hist_resolve, st);
    // AP_ARITH_FAST passes are one-pass rebasing passes: rebase_sample_at reads p.arith
    return launch_formula<TIER, AP_ARITH_REF_CUDA>(p, b, hist_resolve, st);
}

int validate_frame(const ApFrameParams* p, const ApFrameBuffers* b, int hist_resolve) {
    if (!p || !b) {
        set_error("null params or buffers");
        return AP_E_INVALID;
    }
    if (p->width <= 0 || p->height <= 0 || p->factor < 1 || p->max_iter < 0) {
        set_error("bad frame geometry %dx%d factor %d max_iter %d", p->width, p->height, p->factor,
                  p->max_iter);
        return AP_E_INVALID;
    }
    if ((long long)p->width * p->factor > (1LL << 24) || (long long)p->height * p->factor > (1LL << 24)) {
        set_error("sub-sample grid too large");
        return AP_E_INVALID;
    }
    if (p->fractal_type < 0 || p->fractal_type > 4) {
        set_error("fractal_type %d outside 0..4", p->fractal_type);
        return AP_E_INVALID;
    }
    if (p->fractal_type == 4 && (p->gen_n < 0 || p->gen_n > 64)) {
        set_error("gen_n %d outside 0..64", p->gen_n);
        return AP_E_INVALID;
    }
    if (p->tier < AP_TIER_FP64 || p->tier > AP_TIER_FLOATEXP32) {
        set_error("unknown tier %d", p->tier);
        return AP_E_INVALID;
    }
    if (p->arith != AP_ARITH_REF_CPU && p->arith != AP_ARITH_REF_CUDA && p->arith != AP_ARITH_FAST) {
        set_error("unknown arithmetic profile %d", p->arith);
        return AP_E_INVALID;
    }
    if (p->arith == AP_ARITH_FAST && !(p->flags & AP_FLAG_REBASE)) {
        set_error("AP_ARITH_FAST serves one-pass rebasing passes (AP_FLAG_REBASE) only");
        return AP_E_UNSUPPORTED;
    }
    if (p->mode < AP_MODE_COARSE || p->mode > AP_MODE_EDGE) {
        set_error("unknown mode %d", p->mode);
        return AP_E_INVALID;
    }
    if (!b->iter_map) {
        set_error("iter_map is required");
        return AP_E_INVALID;
    }
    if (b->counters && (reinterpret_cast<uintptr_t>(b->counters) & 15u)) {
        set_error("counters must be 16-byte aligned");
        return AP_E_INVALID;
    }
    const bool need_rgb = hist_resolve || p->mode != AP_MODE_COARSE || !(p->flags & AP_FLAG_NO_RGB);
    if (need_rgb && (!b->rgb || !b->lut)) {
        set_error("rgb and lut are required");
        return AP_E_INVALID;
    }
    const bool hist = hist_resolve || (p->flags & AP_FLAG_HIST_COLOUR);
    if (hist && (!b->cdf || p->num_bins < 2)) {
        set_error("histogram colouring needs cdf and num_bins >= 2");
        return AP_E_INVALID;
    }
    if ((p->mode == AP_MODE_EDGE || (hist_resolve && p->rebase_pass == 0)) && !b->edge_mask) {
        set_error("edge_mask is required");
        return AP_E_INVALID;
    }
    if (p->rebase_pass > 0 && !b->glitch_in) {
        set_error("glitch_in is required on rebase passes");
        return AP_E_INVALID;
    }
    if (p->flags & AP_FLAG_REBASE) {
        if (p->tier != AP_TIER_PERTURB && p->tier != AP_TIER_FLOATEXP32) {
            set_error("AP_FLAG_REBASE serves the FP64-delta and FP32 FloatExp tiers (AP_TIER_PERTURB, AP_TIER_FLOATEXP32)");
            return AP_E_UNSUPPORTED;
        }
        if (p->fractal_type == 2 || p->fractal_type == 3) {
            set_error("AP_FLAG_REBASE serves orbits that start at 0 (fractal_type 0, 1, 4)");
            return AP_E_UNSUPPORTED;
        }
        if (p->ref_len < 1 || p->rebase_pass != 0) {
            set_error("AP_FLAG_REBASE needs ref_len >= 1 and rebase_pass 0");
            return AP_E_INVALID;
        }
    }
    if (p->tier >= AP_TIER_PERTURB) {
        if (!b->ref_re || !b->ref_im || p->ref_len < 0) {
            set_error("perturbation tiers need the reference orbit");
            return AP_E_INVALID;
        }
        if (p->bla_levels > 0 && (!b->bla || p->bla_levels > 31)) {
            set_error("bla_levels %d needs a table with at most 31 levels", p->bla_levels);
            return AP_E_INVALID;
        }
    }
    return AP_OK;
}

static int dispatch(const ApFrameParams* p, const ApFrameBuffers* b, int hist_resolve,
                    void* stream) {
    int rc = validate_frame(p, b, hist_resolve);
    if (rc != AP_OK) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (p->tier == AP_TIER_FLOATEXP32) {
        if (hist_resolve) {
            set_error("histogram resolve passes use the FP64 tiers");
            return AP_E_UNSUPPORTED;
        }
        return launch_fe32(*p, *b, st);
    }
    if (!hist_resolve) {
        rc = launch_perturb_fast(*p, *b, st);
        if (rc != AP_E_UNSUPPORTED) return rc;
    }
    switch (p->tier) {
    case AP_TIER_FP64: return launch_arith<AP_TIER_FP64>(*p, *b, hist_resolve, st);
    case AP_TIER_DD: return launch_arith<AP_TIER_DD>(*p, *b, hist_resolve, st);
    case AP_TIER_PERTURB: return launch_arith<AP_TIER_PERTURB>(*p, *b, hist_resolve, st);
    case AP_TIER_FLOATEXP: return launch_arith<AP_TIER_FLOATEXP>(*p, *b, hist_resolve, st);
    default:
        set_error("tier %d is not served by ap_render_pass", p->tier);
        return AP_E_UNSUPPORTED;
    }
}

}  // namespace ap

extern "C" int ap_render_pass(const ApFrameParams* p, const ApFrameBuffers* b, void* stream) {
    return ap::dispatch(p, b, 0, stream);
}

extern "C" int ap_resolve_hist_pass(const ApFrameParams* p, const ApFrameBuffers* b, void* stream) {
    return ap::dispatch(p, b, 1, stream);
}

extern "C" int ap_render_rows(const ApFrameParams* p, const ApFrameBuffers* b, int32_t row0, int32_t rows,
                              void* stream) {
    int rc = ap::validate_frame(p, b, 0);
    if (rc != AP_OK) return rc;
    if (row0 < 0 || rows < 0 || (long long)row0 + rows > p->height) {
        ap::set_error("ap_render_rows: rows [%d, %d) outside the frame's %d rows", row0, row0 + rows, p->height);
        return AP_E_INVALID;
    }
    rc = ap::launch_perturb_fast_rows(*p, *b, row0, rows, static_cast<cudaStream_t>(stream));
    if (rc == AP_E_UNSUPPORTED)
        ap::set_error("ap_render_rows serves coarse AP_TIER_PERTURB passes without in-kernel colour on "
                      "packed inputs (ap_pack_orbit, ap_pack_bla)");
    return rc;
}
