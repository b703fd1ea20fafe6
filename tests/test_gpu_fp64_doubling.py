"""The quadratic step of the CUDA profile with the doubling fused into the sum, fma(2, zx zy, cy) for
(2 zx) zy + cy: the two agree under the rule that admits it (checked in numpy, where 2 (zx zy) is
exact), and device frames on both sides of the rule equal the oracle's bit for bit."""
import ctypes as C

import numpy as np
import pytest

from fractura_b200 import _lib, abi

W, H = 61, 37


def test_the_two_forms_agree_under_the_rule():
    rng = np.random.default_rng(1)
    n = 400000
    mant = lambda: rng.uniform(1, 2, n) * rng.choice([-1.0, 1.0], n)
    ex = rng.integers(-1074, 9, n)                       # |zx| up to the bailout radius
    total = rng.integers(-1090, 18, n)                   # the product's exponent, through the subnormals
    with np.errstate(all="ignore"):
        zx, zy = np.ldexp(mant(), ex), np.ldexp(mant(), np.clip(total - ex, -1074, 9))
        cy = np.ldexp(mant(), rng.integers(-960, 2, n))
        cy[:1000] = np.ldexp(rng.choice([-1.0, 1.0], 1000), -960)
        old, new = (2.0 * zx) * zy + cy, 2.0 * (zx * zy) + cy
        assert np.array_equal(old.view(np.uint64), new.view(np.uint64))
        low = np.ldexp(mant(), -1070)                    # outside the rule they do differ
        assert np.any((2.0 * zx) * zy + low != 2.0 * (zx * zy) + low)
        for c in (0.0, -0.0):                            # cy = zy = 0: zeros of one sign
            for z in (0.0, -0.0):
                old, new = (2.0 * zx) * z + c, 2.0 * (zx * z) + c
                assert np.array_equal(old.view(np.uint64), new.view(np.uint64))


def view(cx, cy, w):
    dx = w / (W - 1)
    return dict(x_min_hi=cx - 0.5 * w, y_max_hi=cy + 0.5 * dx * (H - 1), dx_hi=dx, dy_hi=dx)


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [
    dict(fractal_type=0, **view(-0.75, 0.0, 3.0)), dict(fractal_type=1, **view(-1.7, 0.0, 0.2)),
    dict(fractal_type=0, **view(-1.75, 0.0, 0.1)), dict(fractal_type=0, **view(-1.0, 0.0, 1e-300)),
    dict(fractal_type=2, julia_cx_hi=-1.0, julia_cy_hi=0.0, **view(0.0, 0.0, 1.0)),
    dict(fractal_type=2, julia_cx_hi=-1.0, julia_cy_hi=0.0, **view(0.0, 0.0, 1e-154)),
    dict(fractal_type=2, julia_cx_hi=-1.0, julia_cy_hi=2.0 ** -960, **view(0.0, 0.0, 1e-154)),
    dict(fractal_type=2, julia_cx_hi=-1.0, julia_cy_hi=-(2.0 ** -961), **view(0.0, 0.0, 1e-154)),
    dict(fractal_type=2, julia_cx_hi=-1.9, julia_cy_hi=5e-324, **view(0.0, 0.0, 1e-160)),
    dict(fractal_type=3, julia_cx_hi=-1.0, julia_cy_hi=0.0, **view(0.0, 0.0, 1e-154)),
    dict(fractal_type=2, julia_cx_hi=-0.8, julia_cy_hi=0.156, **view(0.0, 0.0, 3.0))])
def test_frames_on_both_sides_of_the_rule(kw):
    import oracle
    import torch
    p = abi.new_params(width=W, height=H, factor=1, tier=abi.AP_TIER_FP64, arith=abi.AP_ARITH_REF_CUDA, mode=abi.AP_MODE_COARSE,
                       flags=abi.AP_FLAG_NO_RGB, max_iter=700, **kw)
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
