"""FloatExp frames of z^2 + c, whose late steps run on the delta itself: equal to the oracle's, which
scales every step, bit for bit -- spirals with their leaps, a view centred on the real axis (a
component that stays zero), bounded pixels, glitch tests on and off, Julia sets, odd frame sizes."""
from decimal import Decimal

import numpy as np
import pytest

from fractura_b200 import engine
from fractura_b200 import high_precision as hp
from helpers import oracle_pert_frame
from test_gpu_fexp import META

pytestmark = pytest.mark.gpu
BASE = next(x for x in META if x["name"] == "fexp_mandel")


@pytest.mark.parametrize("arith", ["ref_cpu", "ref_cuda"])
@pytest.mark.parametrize("glitch", ["Off (Single-Ref)", "Pauldelbrot"])
@pytest.mark.parametrize("ft,cx,cy,width,max_iter", [
    (0, "0", "1", "1e-305", 3000), (0, "0", "1", "1e-1000", 4000), (0, "-2", "0", "1e-400", 1500),
    (0, "-1", "0", "1e-301", 400), (0, "0.25", "0", "1e-310", 500),
    (0, "-1.5436890126920763615708559718017479865252032976509835527", "0", "1e-320", 900),
    (2, "0", "0", "1e-305", 300), (2, "1.6180339887498948482", "0", "1e-330", 600)])
def test_frames_equal_the_oracle(ft, cx, cy, width, max_iter, glitch, arith):
    W, H = 47, 29
    m = dict(BASE, W=W, H=H, cx=cx, cy=cy, width=width, max_iter=max_iter, fractal_type=ft, julia_cx=-1.0, julia_cy=0.0,
             factor=1, scheme=0, bbsa_order=32, glitch_mode=glitch)
    hp.clear_reference_orbit_cache()
    it = np.zeros((H, W), np.float32)
    engine.render_frame_ssaa(
        W, H, max_iter, Decimal(cx), Decimal(cy), Decimal(width), None, color_scheme_id=0,
        precision_mode="1e-300 (Perturbation)", fractal_type=ft, julia_cx=-1.0, julia_cy=0.0, bbsa_tol=1e-6,
        bbsa_order=32, glitch_mode=glitch, gen_n=m["gen_n"], gen_kr=m["gen_kr"], gen_ki=m["gen_ki"], h_iter_buf=it,
        arith=arith)
    fr, _ = oracle_pert_frame(m, arith=0 if arith == "ref_cpu" else 1)
    assert np.array_equal(it.view(np.uint32), fr.iter_map.view(np.uint32)), \
        int((it.view(np.uint32) != fr.iter_map.view(np.uint32)).sum())
