"""FP64 direct iteration in blocks of untested steps with cycle detection: device frames equal the
oracle's, which tests every step and iterates bounded pixels to the end, bit for bit -- at depths
around the lead and block lengths, with bounded regions, and where blocks are not allowed (large
|c|, Multibrot n < 2 or large k)."""
import ctypes as C

import numpy as np
import pytest

from fractura_b200 import _lib, abi

pytestmark = pytest.mark.gpu
W, H = 61, 37


def compare(arith=abi.AP_ARITH_REF_CPU, **kw):
    import oracle
    import torch
    p = abi.new_params(width=W, height=H, factor=1, tier=abi.AP_TIER_FP64, arith=arith, mode=abi.AP_MODE_COARSE,
                       flags=abi.AP_FLAG_NO_RGB, **kw)
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
    return fr


def view(cx, cy, w):
    dx = w / (W - 1)
    return dict(x_min_hi=cx - 0.5 * w, y_max_hi=cy + 0.5 * dx * (H - 1), dx_hi=dx, dy_hi=dx)


@pytest.mark.parametrize("max_iter", [0, 1, 7, 8, 9, 23, 24, 25, 26, 39, 40, 41, 56, 57])
@pytest.mark.parametrize("ft", [0, 3, 4])
def test_depths_around_the_block_lengths(ft, max_iter):
    compare(max_iter=max_iter, fractal_type=ft, julia_cx_hi=-1.755, julia_cy_hi=0.03, gen_n=3, gen_kr=0.1, gen_ki=0.2,
            **view(-0.5, 0.0, 3.2))


@pytest.mark.parametrize("arith", [abi.AP_ARITH_REF_CPU, abi.AP_ARITH_REF_CUDA])
@pytest.mark.parametrize("ft,n", [(0, 2), (1, 2), (2, 2), (3, 2), (4, 2), (4, 3), (4, 4), (4, 5), (4, 7)])
def test_bounded_regions(ft, n, arith):
    fr = compare(arith, max_iter=20000, fractal_type=ft, julia_cx_hi=-0.12, julia_cy_hi=0.6, gen_n=n, gen_kr=0.1,
                 gen_ki=0.2, **view(-0.3, 0.0, 3.0))
    assert np.count_nonzero(fr.kmap == -1) > 10


@pytest.mark.parametrize("kw", [
    dict(fractal_type=0, **view(0.0, 0.0, 5000.0)), dict(fractal_type=1, **view(-990.0, 990.0, 40.0)),
    dict(fractal_type=2, julia_cx_hi=1500.0, julia_cy_hi=0.1, **view(0.0, 0.0, 100.0)),
    dict(fractal_type=4, gen_n=0, gen_kr=0.5, gen_ki=0.1, **view(0.0, 0.0, 4.0)),
    dict(fractal_type=4, gen_n=1, gen_kr=-0.9, gen_ki=0.1, **view(0.0, 0.0, 4.0)),
    dict(fractal_type=4, gen_n=2, gen_kr=300.0, gen_ki=0.0, **view(0.0, 0.0, 4.0)),
    dict(fractal_type=2, julia_cx_hi=0.1, julia_cy_hi=0.0, **view(1e160, 0.0, 1e160))])
def test_where_blocks_are_not_allowed(kw):
    compare(max_iter=300, **kw)
