"""Supersampling passes deal single samples to lanes: frames equal the oracle's, whose pixels take their
samples one after the other, where a pixel's samples fill part of a warp's round, exactly one, or
several, and where the frame ends inside a patch."""
from decimal import Decimal

import numpy as np
import pytest

from fractura_b200 import abi, engine
from fractura_b200 import high_precision as hp
from helpers import oracle_pert_frame
from test_gpu_direct import check_against_oracle

pytestmark = pytest.mark.gpu
BASE = dict(cx="-0.7436", cy="0.1318", width="0.02", fractal_type=0, julia_cx=-0.8, julia_cy=0.156, gen_n=3,
            gen_kr=0.25, gen_ki=1.0, offset=0.1, density=1.0, contrast=1.0, max_iter=300)


@pytest.mark.parametrize("factor", [2, 3, 6, 7])
@pytest.mark.parametrize("W,H", [(8, 4), (33, 9), (61, 22)])
@pytest.mark.parametrize("scheme", [2, 11])
@pytest.mark.parametrize("arith,code", [("ref_cpu", abi.AP_ARITH_REF_CPU), ("ref_cuda", abi.AP_ARITH_REF_CUDA)])
def test_direct_frames(factor, W, H, scheme, arith, code):
    m = dict(BASE, W=W, H=H, factor=factor, scheme=scheme)
    check_against_oracle(m, abi.AP_TIER_FP64, arith, code)
    if factor < 6:
        check_against_oracle(dict(m, width="1e-13"), abi.AP_TIER_DD, arith, code)


@pytest.mark.parametrize("factor", [2, 3, 6])
@pytest.mark.parametrize("glitch", ["Off (Single-Ref)", "Pauldelbrot"])
@pytest.mark.parametrize("width", ["1e-14", "1e-320"])
def test_perturbation_frames(factor, glitch, width):
    deep = dict(cx="0.0", cy="1.0") if width == "1e-320" else {}
    m = dict({**BASE, **deep}, W=29, H=13, factor=factor, scheme=0, width=width, max_iter=1500, bbsa_order=32,
             glitch_mode=glitch, offset=0.0)
    it = np.zeros((13, 29), np.float32)
    hp.clear_reference_orbit_cache()
    rgb = engine.render_frame_ssaa(29, 13, 1500, Decimal(m["cx"]), Decimal(m["cy"]), Decimal(width), None,
                                   ssaa_factor=factor, color_scheme_id=0, precision_mode="1e-300 (Perturbation)",
                                   bbsa_tol=1e-6, bbsa_order=32, glitch_mode=glitch, h_iter_buf=it)
    fr, _ = oracle_pert_frame(m)
    assert np.array_equal(it.view(np.uint32), fr.iter_map.view(np.uint32))
    assert np.array_equal(rgb, fr.rgb)


@pytest.mark.parametrize("factor", [2, 3])
def test_glitch_map_in_place(factor):
    """A rebase pass that writes its glitches into the map that chose its pixels equals one with two maps."""
    import ctypes as C

    import torch
    from fractura_b200 import _lib
    from fractura_b200.palette import synthetic_lut
    from helpers import load_golden
    from test_oracle_fexp import floatexp_params
    G, META = load_golden("fexp_samples.npz")
    m = next(x for x in META if x["name"] == "fexp_mandel")
    _, p = floatexp_params(m, "plain", abi.AP_ARITH_REF_CUDA)
    W, H = 61, 22
    p.width, p.height, p.factor, p.mode, p.rebase_pass = W, H, factor, abi.AP_MODE_FULL, 1
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    re, im, lut = dev(G["fexp_mandel__re"]), dev(G["fexp_mandel__im"]), dev(synthetic_lut())
    marks = (np.random.default_rng(factor).random((H, W)) < 0.8).astype(np.uint8)
    got = []
    for same in (False, True):
        gin, it = dev(marks), torch.zeros((H, W), dtype=torch.float32, device="cuda")
        gout = gin if same else dev(marks)
        rgb = torch.zeros((H, W, 3), dtype=torch.uint8, device="cuda")
        b = abi.ApFrameBuffers()
        ptr = lambda x: C.c_void_p(x.data_ptr())
        b.ref_re, b.ref_im, b.lut, b.iter_map, b.rgb = ptr(re), ptr(im), ptr(lut), ptr(it), ptr(rgb)
        b.glitch_in, b.glitch_out = ptr(gin), ptr(gout)
        _lib.check(_lib.load().ap_render_pass(C.byref(p), C.byref(b), None), "ap_render_pass")
        got.append((rgb.cpu().numpy(), gout.cpu().numpy()))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert got[0][0].any()
