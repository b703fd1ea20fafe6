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
