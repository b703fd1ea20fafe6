"""The double-double step's short sums: equal to the general ones on normalised operands
(CPU, the formulas restated in numpy), and device frames equal the oracle's where the
step changes path: zero rows, tiny and unnormalised values, values near the bailout."""
import ctypes as C

import numpy as np
import pytest

from fractura_b200 import _lib, abi


def two_sum(a, b):
    s = a + b
    v = s - a
    return s, (a - (s - v)) + (b - v)


def quick_sum(a, b):
    s = a + b
    return s, b - (s - a)


def random_dd(rng, n, exp):
    hi = rng.uniform(1.0, 2.0, n) * rng.choice([-1.0, 1.0], n) * np.exp2(exp)
    lo = np.spacing(np.abs(hi)) * rng.uniform(-0.5, 0.5, n)
    lo[rng.random(n) < 0.1] = 0.0
    return two_sum(hi, lo)


@pytest.mark.parametrize("seed", range(4))
def test_quick_second_sum_equals_the_general_one(seed):
    """dd_add's second sum, for operands of any relation: far apart, equal, cancelling to a few ulps."""
    rng = np.random.default_rng(seed)
    n = 200_000
    ah, al = random_dd(rng, n, rng.integers(-3, 4, n))
    bh, bl = random_dd(rng, n, rng.integers(-60, 4, n))
    near = rng.random(n) < 0.6  # b close to -a: a few ulps off, or exactly opposite
    ch = -ah + np.spacing(ah) * rng.integers(-3, 4, n)
    ch = np.where(rng.random(n) < 0.3, -ah, ch)
    cl = np.spacing(np.abs(ch)) * rng.uniform(-0.5, 0.5, n)
    ch, cl = two_sum(ch, cl)
    bh, bl = np.where(near, ch, bh), np.where(near, cl, bl)
    sh, sl = two_sum(ah, bh)
    t = (sl + al) + bl
    want, got = two_sum(sh, t), quick_sum(sh, t)
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])


CASES = {  # x_min, y_max, dx, dy as (hi, lo), Julia constant as (hi, lo) pairs
    "zero row and column": ((-1.0, 0.0), (0.5, 0.0), (2.0 / 32, 0.0), (1.0 / 16, 0.0), (0.0, 0.0), (0.0, 0.0)),
    "around 2^-200": ((-16 * 2.0 ** -203, 0.0), (8 * 2.0 ** -203, 0.0), (2.0 ** -203, 0.0), (2.0 ** -203, 0.0),
                      (-0.8, 2.0 ** -710), (0.156, 0.0)),
    "tiny low parts": ((-0.75, 2.0 ** -720), (0.1, 2.0 ** -690), (2.0 ** -9, 2.0 ** -730), (2.0 ** -9, 2.0 ** -700),
                       (-0.4, 2.0 ** -720), (0.6, 0.0)),
    "unnormalised constant": ((-1.2, 0.0), (0.7, 0.0), (2.4 / 32, 0.0), (1.4 / 16, 0.0), (0.25, 0.035), (0.0, 0.01)),
    "near the bailout": ((-300.0, 0.0), (280.0, 1e-20), (600.0 / 32, 0.0), (560.0 / 16, 0.0), (-200.5, 0.0), (3.0, 0.0)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("arith", [abi.AP_ARITH_REF_CPU, abi.AP_ARITH_REF_CUDA])
@pytest.mark.parametrize("ft", [0, 1, 2, 3])
@pytest.mark.parametrize("case", sorted(CASES))
def test_device_equals_oracle_where_the_step_changes_path(case, ft, arith):
    import oracle
    import torch
    (xh, xl), (yh, yl), (dxh, dxl), (dyh, dyl), (jx, jxl), (jy, jyl) = CASES[case]
    W, H = 33, 17
    p = abi.new_params(width=W, height=H, factor=1, max_iter=200, fractal_type=ft, tier=abi.AP_TIER_DD, arith=arith,
                       mode=abi.AP_MODE_COARSE, flags=abi.AP_FLAG_NO_RGB, x_min_hi=xh, x_min_lo=xl, y_max_hi=yh,
                       y_max_lo=yl, dx_hi=dxh, dx_lo=dxl, dy_hi=dyh, dy_lo=dyl, julia_cx_hi=jx, julia_cx_lo=jxl,
                       julia_cy_hi=jy, julia_cy_lo=jyl)
    fr = oracle.Frame(W, H)
    oracle.render_pass(p, fr)
    it = torch.empty((H, W), dtype=torch.float32, device="cuda")
    km = torch.empty((H, W), dtype=torch.int32, device="cuda")
    b = abi.ApFrameBuffers()
    b.iter_map, b.kmap = C.c_void_p(it.data_ptr()), C.c_void_p(km.data_ptr())
    _lib.check(_lib.load().ap_render_pass(C.byref(p), C.byref(b), C.c_void_p(torch.cuda.current_stream().cuda_stream)),
               "ap_render_pass")
    assert np.array_equal(km.cpu().numpy(), fr.kmap)
    assert np.array_equal(it.cpu().numpy().view(np.uint32), fr.iter_map.view(np.uint32))


def plain_range(parts, top=0x4066a000):
    """PlainRange of ap_dd.cuh on columns (x.hi, y.hi, x.lo, y.lo): high words, unsigned."""
    h = [(p.view(np.uint64) >> np.uint64(32)).astype(np.uint32) & np.uint32(0x7fffffff) for p in parts]
    high = np.minimum(h[0] - np.uint32(1), h[1] - np.uint32(1))
    low = np.minimum(h[2] - np.uint32(1), h[3] - np.uint32(1))
    return ((np.maximum(h[0], h[1]) < top) & (high >= ((1023 - 200) << 20) - 1) & (low >= ((1023 - 700) << 20) - 1))


def test_range_words_are_the_ranges_they_stand_for():
    """Both edges of each range, zeros of both signs, infinities and NaN of both signs, in every part.  (Numbers below
    2^-1042, whose high word is 0, count as 0.)"""
    inf, nan = np.inf, np.nan
    edges = [0.0, 2.0 ** -1042, 2.0 ** -1000, 2.0 ** -700, np.nextafter(2.0 ** -700, 0), 2.0 ** -200,
             np.nextafter(2.0 ** -200, 0), 1.0, 2.0, np.nextafter(181.0, 0), 181.0, 256.0, 1e300, inf, nan]
    v = np.array(edges + [-e for e in edges])
    grid = [g.ravel().copy() for g in np.meshgrid(v, v, v, v)]
    with np.errstate(invalid="ignore"):
        a = np.abs(np.array(grid))
        want = np.ones(a.shape[1], bool)
        for q in (0, 1):
            want &= (a[q] < 181.0) & ((a[q] == 0.0) | (a[q] >= 2.0 ** -200))
        for q in (2, 3):
            want &= (a[q] == 0.0) | (a[q] >= 2.0 ** -700) | np.isnan(a[q])  # a NaN low part has a NaN high one
    assert np.array_equal(plain_range(grid), want)
    with np.errstate(invalid="ignore"):  # finite(): up to 2^400
        for q in (0, 1):
            grid[q][a[q] == 1e300] = 2.0 ** 400
            grid[q][a[q] == 256.0] = np.nextafter(2.0 ** 400, 0)
        a = np.abs(np.array(grid))
        want = np.ones(a.shape[1], bool)
        for q in (0, 1):
            want &= (a[q] < 2.0 ** 400) & ((a[q] == 0.0) | (a[q] >= 2.0 ** -200))
        for q in (2, 3):
            want &= (a[q] == 0.0) | (a[q] >= 2.0 ** -700) | np.isnan(a[q])
    assert np.array_equal(plain_range(grid, (1023 + 400) << 20), want)


@pytest.mark.gpu
@pytest.mark.parametrize("arith", [abi.AP_ARITH_REF_CPU, abi.AP_ARITH_REF_CUDA])
@pytest.mark.parametrize("ft", [0, 1, 2])
@pytest.mark.parametrize("max_iter", [0, 1, 31, 32, 33, 39, 40, 41, 48, 203])
def test_depths_that_end_anywhere_in_a_block(max_iter, ft, arith):
    """The whole sets (escapes at every place of a block, a zero row, bounded pixels)."""
    import oracle
    import torch
    W, H = 41, 33
    p = abi.new_params(width=W, height=H, factor=1, max_iter=max_iter, fractal_type=ft, tier=abi.AP_TIER_DD, arith=arith,
                       mode=abi.AP_MODE_COARSE, flags=abi.AP_FLAG_NO_RGB, x_min_hi=-2.1, x_min_lo=1e-18, y_max_hi=1.5,
                       dx_hi=3.2 / 40, dy_hi=3.0 / 32, julia_cx_hi=-0.8, julia_cx_lo=1e-20, julia_cy_hi=0.156)
    fr = oracle.Frame(W, H)
    oracle.render_pass(p, fr)
    it = torch.empty((H, W), dtype=torch.float32, device="cuda")
    km = torch.empty((H, W), dtype=torch.int32, device="cuda")
    b = abi.ApFrameBuffers()
    b.iter_map, b.kmap = C.c_void_p(it.data_ptr()), C.c_void_p(km.data_ptr())
    _lib.check(_lib.load().ap_render_pass(C.byref(p), C.byref(b), C.c_void_p(torch.cuda.current_stream().cuda_stream)),
               "ap_render_pass")
    assert np.array_equal(km.cpu().numpy(), fr.kmap)
    assert np.array_equal(it.cpu().numpy().view(np.uint32), fr.iter_map.view(np.uint32))
