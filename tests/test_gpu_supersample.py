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
