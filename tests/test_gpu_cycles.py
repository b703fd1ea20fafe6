"""Cycle detection of the packed perturbation kernels (one-pass rebasing and one reference): bounded
pixels whose state repeats skip whole cycles, and every output stays what iterating them to max_iter
gives (the oracle), bit for bit -- with and without leaps, at depths that end anywhere in a cycle,
per frame and in the batch kernel at a quantum of one step."""
import ctypes as C
import json
import os
from decimal import Decimal

import numpy as np
import pytest

from fractura_b200 import abi, engine
from fractura_b200 import batch as fb
from fractura_b200 import high_precision as hp
from fractura_b200.perturbation import ONE_PASS_REBASING
from helpers import GOLDEN, oracle_pert_frame

pytestmark = pytest.mark.gpu
ARITH = {"ref_cpu": abi.AP_ARITH_REF_CPU, "ref_cuda": abi.AP_ARITH_REF_CUDA, "fast": abi.AP_ARITH_FAST}


def _views():
    with open(os.path.join(GOLDEN, "workloads.json")) as f:
        tiles = json.load(f)["config4_tiles"]
    keys = ("cx", "cy", "width", "fractal_type", "julia_cx", "julia_cy", "gen_n", "gen_kr", "gen_ki")
    out = {f"tile{q}": dict({k: tiles[q][k] for k in keys}, max_iter=mi)
           for q, mi in ((3, 6007), (10, 3000), (13, 4001), (17, 3738), (22, 5003))}
    plain = dict(julia_cx=0.0, julia_cy=0.0, gen_n=3, gen_kr=0.25, gen_ki=1.0)
    # beside and inside the period-3 disc: the reference settles on its cycle
    out["mandel"] = dict(plain, cx="-0.1226", cy="0.7449", width="1e-13", fractal_type=0, max_iter=2500)
    out["julia"] = dict(plain, cx="0.05", cy="0.02", width="1e-13", fractal_type=2, julia_cx=-0.12, julia_cy=0.6,
                        max_iter=2501)
    return out


VIEWS = _views()


def frame(m, arith, glitch, bla_form):
    import torch
    W, H = m["W"], m["H"]
    kmap = torch.empty((H, W), dtype=torch.int32, device="cuda")
    it = np.zeros((H, W), np.float32)
    hp.clear_reference_orbit_cache()
    engine.render_frame_ssaa(W, H, m["max_iter"], Decimal(m["cx"]), Decimal(m["cy"]), Decimal(m["width"]), None,
                             color_scheme_id=0, precision_mode="1e-300 (Perturbation)", fractal_type=m["fractal_type"],
                             julia_cx=m["julia_cx"], julia_cy=m["julia_cy"], bbsa_tol=1e-6, bbsa_order=m["bbsa_order"],
                             glitch_mode=glitch, gen_n=m["gen_n"], gen_kr=m["gen_kr"], gen_ki=m["gen_ki"], h_iter_buf=it,
                             arith=arith, bla_form=bla_form, _extra_out=(kmap, None))
    return it, kmap.cpu().numpy()


@pytest.mark.parametrize("order,bla_form", [(0, "reference"), (32, "accurate"), (32, "reference")])
@pytest.mark.parametrize("arith,glitch", [("fast", ONE_PASS_REBASING), ("ref_cpu", ONE_PASS_REBASING),
                                          ("ref_cuda", "Off (Single-Ref)"), ("ref_cpu", "Off (Single-Ref)")])
@pytest.mark.parametrize("name", sorted(VIEWS))
def test_frames_equal_the_oracle(name, arith, glitch, order, bla_form):
    v = VIEWS[name]
    if glitch == ONE_PASS_REBASING and v["fractal_type"] == 2:
        pytest.skip("Julia orbits do not rebase")
    m = dict(v, W=23, H=17, factor=1, scheme=0, bbsa_order=order, bbsa_tol=1e-6, glitch_mode=glitch)
    it, k = frame(m, arith, glitch, bla_form)
    fr, _ = oracle_pert_frame(m, arith=ARITH[arith],
                              bla_eps=engine.ACCURATE_BLA_EPS if bla_form == "accurate" else None)
    assert np.count_nonzero(fr.kmap == -1) > 0
    assert np.array_equal(k, fr.kmap)
    assert np.array_equal(it.view(np.uint32), fr.iter_map.view(np.uint32))


@pytest.mark.parametrize("quantum", [1, 37, 256])
def test_batch_skips_cycles_with_the_frames_values(quantum):
    import torch
    hp.clear_reference_orbit_cache()
    tiles = [fb.Tile(cx=Decimal(v["cx"]), cy=Decimal(v["cy"]), width=Decimal(v["width"]), W=23, H=17,
                     max_iter=v["max_iter"], fractal_type=v["fractal_type"], julia_cx=v["julia_cx"],
                     julia_cy=v["julia_cy"], gen_n=v["gen_n"], gen_kr=v["gen_kr"], gen_ki=v["gen_ki"],
                     strict_glitch=False, rebase=v["fractal_type"] != 2) for v in VIEWS.values()]
    b = fb.prepare_batch(tiles, arith="ref_cpu", bla_form="accurate")
    work = [torch.zeros((t.H, t.W, 4), dtype=torch.int32, device="cuda") for t in tiles]
    for slot, q in enumerate(b.order):
        b.desc_host[slot].counters = C.c_void_p(work[q].data_ptr())
    b.desc_dev = torch.from_numpy(np.frombuffer(bytes(b.desc_host), dtype=np.uint8).copy()).cuda()
    b.render(fb.BatchConfig(quantum=quantum))
    torch.cuda.synchronize()
    for name, t, out, w in zip(VIEWS, tiles, b.tiles_out, work):
        m = dict(VIEWS[name], W=t.W, H=t.H, factor=1, scheme=0, bbsa_order=32)
        it, k = frame(m, "ref_cpu", ONE_PASS_REBASING if t.rebase else "Off (Single-Ref)", "accurate")
        assert np.array_equal(out["kmap"].cpu().numpy(), k)
        assert np.array_equal(out["iter"].cpu().numpy().view(np.uint32), it.view(np.uint32))
        c = w.cpu().numpy()
        assert c.min() >= 0 and np.all(c[..., 0] <= t.max_iter)
        if name in ("tile10", "tile13"):  # bounded pixels of these settle within 2500 steps
            assert c[k == -1][:, 0].mean() < 0.9 * t.max_iter
