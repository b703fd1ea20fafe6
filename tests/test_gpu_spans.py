"""Runs of untested steps (AP_FLAG_SPANS): frames equal the oracle's, which tests every step, bit for
bit -- where the leap radii are wide, where dc is not negligible beside the delta, for Julia deltas
that start at dc, without leaps, and past the reference's end, where z is iterated in blocks."""
from decimal import Decimal

import numpy as np
import pytest

import oracle
from fractura_b200 import abi, engine
from fractura_b200 import high_precision as hp
from fractura_b200.perturbation import ONE_PASS_REBASING
from helpers import oracle_pert_frame

pytestmark = pytest.mark.gpu
ARITH = {"ref_cpu": abi.AP_ARITH_REF_CPU, "ref_cuda": abi.AP_ARITH_REF_CUDA, "fast": abi.AP_ARITH_FAST}
PLAIN = dict(julia_cx=0.0, julia_cy=0.0, gen_n=3, gen_kr=0.25, gen_ki=1.0)
SEAHORSE = dict(PLAIN, cx="-0.743643887037158704752191506114774", cy="0.131825904205311970493132056385139",
                fractal_type=0)
VIEWS = {
    "1e-13": dict(SEAHORSE, width="9e-13", max_iter=3000),
    "1e-26": dict(SEAHORSE, width="1e-26", max_iter=20000),
    "spiral": dict(PLAIN, cx="0.0", cy="1.0", width="1e-40", fractal_type=0, max_iter=2000),
    "julia": dict(PLAIN, cx="0.0000001", cy="0.3", width="5e-13", fractal_type=2, julia_cx=-0.8, julia_cy=0.156,
                  max_iter=3000),
    "multibrot": dict(PLAIN, cx="0.35", cy="-0.55", width="8e-13", fractal_type=4, max_iter=1500),
}


@pytest.mark.parametrize("order,tol,bla_form", [(0, 0.0, "reference"), (32, 1e-4, "reference"),
                                                (32, 3e-2, "reference"), (32, 1e-6, "accurate")])
@pytest.mark.parametrize("arith,glitch", [("fast", ONE_PASS_REBASING), ("ref_cuda", ONE_PASS_REBASING),
                                          ("ref_cpu", "Off (Single-Ref)"), ("ref_cuda", "Pauldelbrot")])
@pytest.mark.parametrize("name", sorted(VIEWS))
def test_frames_equal_the_oracle(name, arith, glitch, order, tol, bla_form, monkeypatch):
    import torch
    # the oracle's frames build the reference table at 1e-6: here at the case's tolerance
    build = oracle.build_bla
    monkeypatch.setattr(oracle, "build_bla", lambda re, im, rl, ft, _, *rest: build(re, im, rl, ft, tol, *rest))
    v = VIEWS[name]
    if glitch == ONE_PASS_REBASING and v["fractal_type"] == 2:
        pytest.skip("Julia orbits do not rebase")
    m = dict(v, W=31, H=19, factor=1, scheme=0, bbsa_order=order, bbsa_tol=tol, glitch_mode=glitch)
    kmap = torch.empty((19, 31), dtype=torch.int32, device="cuda")
    it = np.zeros((19, 31), np.float32)
    hp.clear_reference_orbit_cache()
    engine.render_frame_ssaa(31, 19, m["max_iter"], Decimal(m["cx"]), Decimal(m["cy"]), Decimal(m["width"]), None,
                             color_scheme_id=0, precision_mode="1e-300 (Perturbation)", fractal_type=m["fractal_type"],
                             julia_cx=m["julia_cx"], julia_cy=m["julia_cy"], bbsa_tol=tol, bbsa_order=order,
                             glitch_mode=glitch, gen_n=m["gen_n"], gen_kr=m["gen_kr"], gen_ki=m["gen_ki"], h_iter_buf=it,
                             arith=arith, bla_form=bla_form, _extra_out=(kmap, None))
    fr, _ = oracle_pert_frame(m, arith=ARITH[arith],
                              bla_eps=engine.ACCURATE_BLA_EPS if bla_form == "accurate" else None)
    assert np.array_equal(kmap.cpu().numpy(), fr.kmap)
    assert np.array_equal(it.view(np.uint32), fr.iter_map.view(np.uint32))
