"""The forms of the packed coarse pass -- spans or not (a rule on the leaps' tolerance; without leaps
always), the periodic tail's visits or not (the orbit's own) -- give the same maps, bit for bit, per
frame and in a batch."""
from decimal import Decimal

import numpy as np
import pytest

from fractura_b200 import batch as fb
from fractura_b200 import engine, perturbation
from fractura_b200 import high_precision as hp
from fractura_b200.perturbation import ONE_PASS_REBASING


def test_spans_rule():
    assert all(perturbation.spans_allowed(ft, t) for ft in (0, 2) for t in (1e-14, 1e-10))
    assert not any(perturbation.spans_allowed(ft, t) for ft in (0, 2) for t in (0.0, -1.0, 1.1e-10, 1e-6, float("nan")))
    assert not any(perturbation.spans_allowed(ft, 1e-14) for ft in (1, 3, 4))
    assert perturbation.spans_allowed(0, 1e-4, loosest=1e-4) and not perturbation.spans_allowed(0, 1.1e-4, loosest=1e-4)


VIEWS = {  # an escaping reference, a bounded one without a tail, one with a tail
    "escaping": dict(cx="-0.743643887037158704752191506114774", cy="0.131825904205311970493132056385139", width="1e-22", max_iter=20000),
    "long": dict(cx="-0.743643887037158704752191506114774", cy="0.131825904205311970493132056385139", width="1e-26", max_iter=9000),
    "tail": dict(cx="-0.1226", cy="0.7449", width="1e-13", max_iter=2500),
}


def _frame(v, tol, glitch, arith):
    import torch
    W, H = 37, 19
    k = torch.empty((H, W), dtype=torch.int32, device="cuda")
    s = torch.empty((H, W), dtype=torch.float64, device="cuda")
    hp.clear_reference_orbit_cache()
    engine.render_frame_ssaa(W, H, v["max_iter"], Decimal(v["cx"]), Decimal(v["cy"]), Decimal(v["width"]), None,
                             color_scheme_id=0, precision_mode="1e-300 (Perturbation)", bbsa_tol=tol, bbsa_order=32,
                             glitch_mode=glitch, arith=arith, bla_form="reference", _extra_out=(k, s))
    return k.cpu().numpy(), s.cpu().numpy().view(np.uint64)


@pytest.mark.gpu
@pytest.mark.parametrize("tol", [1e-5, 1e-9, 1e-10, 1e-13])
@pytest.mark.parametrize("arith,glitch", [("fast", ONE_PASS_REBASING), ("ref_cpu", ONE_PASS_REBASING),
                                          ("ref_cuda", "Off (Single-Ref)"), ("ref_cpu", "Off (Single-Ref)")])
@pytest.mark.parametrize("name", sorted(VIEWS))
def test_frames_with_and_without_spans(name, arith, glitch, tol, monkeypatch):
    out = []
    for on in (False, True):
        monkeypatch.setattr(perturbation, "spans_allowed", lambda *a, on=on, **kw: on)
        out.append(_frame(VIEWS[name], tol, glitch, arith))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.gpu
@pytest.mark.parametrize("arith", ["ref_cpu", "ref_cuda"])
@pytest.mark.parametrize("dx", [0.0, 1e-300, 1e-26, 1e-9, 1e-3, float("nan"), float("inf")])
@pytest.mark.parametrize("z0", [0.0, 1e-305, 1e-30, 1e-8, 1e-2])
def test_spans_without_leaps_against_the_oracle(z0, dx, arith):
    """Deltas far below dc, far above it, zero, subnormal in the square, and not finite: a Julia view (the delta starts
    at the pixel: z0 wide, with an offset of its own) and a Mandelbrot one (it starts at 0, dc = dx wide)."""
    import ctypes as C

    import oracle
    import torch
    from fractura_b200 import _lib, abi
    n, W, H = 300, 9, 5
    L = _lib.load()
    for ft, d in ((2, z0), (0, dx)):
        z, o = (0.0 if ft == 0 else 0.3 + 0.2j), []
        for _ in range(n + 1):
            o.append(complex(z))
            z = z * z + (-0.12 + 0.6j if ft == 2 else -0.5 + 0.5j)
        re, im = np.array([v.real for v in o]), np.array([v.imag for v in o])
        p = abi.new_params(width=W, height=H, max_iter=350, fractal_type=ft, tier=abi.AP_TIER_PERTURB, dx_hi=d, dy_hi=d,
                           arith=getattr(abi, "AP_ARITH_" + arith.upper()), ref_px=1.5, ref_py=2.25, ref_len=n, julia_cx_hi=-0.12,
                           julia_cy_hi=0.6, ref_cx=-0.5, ref_cy=0.5, strict_glitch=1, flags=abi.AP_FLAG_NO_RGB)
        _, want_g, want_k, want_s = oracle.pert_grid(p, re, im, None, np.arange(W, dtype=np.float64),
                                                     np.arange(H, dtype=np.float64), with_s64=True)
        t = [torch.from_numpy(a).cuda() for a in (re, im)]
        po = torch.zeros((n + 1) * 6, dtype=torch.float64, device="cuda")
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(L.ap_pack_orbit(C.c_void_p(t[0].data_ptr()), C.c_void_p(t[1].data_ptr()), n, C.c_void_p(po.data_ptr()), st),
                   "ap_pack_orbit")
        it = torch.empty((H, W), dtype=torch.float32, device="cuda")
        k = torch.empty((H, W), dtype=torch.int32, device="cuda")
        s = torch.empty((H, W), dtype=torch.float64, device="cuda")
        g = torch.empty((H, W), dtype=torch.uint8, device="cuda")
        b = abi.ApFrameBuffers()
        b.ref_re, b.ref_im, b.orbit_packed = (C.c_void_p(v.data_ptr()) for v in (*t, po))
        b.iter_map, b.kmap, b.s64, b.glitch_out = (C.c_void_p(v.data_ptr()) for v in (it, k, s, g))
        _lib.check(L.ap_render_pass(C.byref(p), C.byref(b), st), "ap_render_pass")
        assert np.array_equal(k.cpu().numpy(), want_k) and np.array_equal(g.cpu().numpy() != 0, want_g != 0)
        assert np.array_equal(s.cpu().numpy(), want_s, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("arith", ["fast", "ref_cpu"])
def test_batch_with_and_without_spans(arith, monkeypatch):
    import torch
    out = []
    for on in (False, True):
        monkeypatch.setattr(perturbation, "spans_allowed", lambda *a, on=on, **kw: on)
        hp.clear_reference_orbit_cache()
        tiles = [fb.Tile(cx=Decimal(v["cx"]), cy=Decimal(v["cy"]), width=Decimal(v["width"]), W=37, H=19, max_iter=v["max_iter"],
                         fractal_type=0, strict_glitch=False, rebase=rebase) for v in VIEWS.values() for rebase in (True, False)]
        b = fb.prepare_batch(tiles, arith=arith, bla_form="accurate")
        b.render()
        torch.cuda.synchronize()
        out.append([(o["kmap"].cpu().numpy(), o["iter"].cpu().numpy().view(np.uint32)) for o in b.tiles_out])
    assert all(np.array_equal(x, y) for p, q in zip(*out) for x, y in zip(p, q))
