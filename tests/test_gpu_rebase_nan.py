"""One-pass rebasing with deltas that are not numbers: such a pixel ends at once, flagged, as the
oracle ends it -- with infinite and NaN spacings, and with a Multibrot coefficient whose products
overflow -- and the high-word test that this rests on holds for NaN of either sign."""
import ctypes as C

import numpy as np
import pytest

from fractura_b200 import _lib, abi


def _high(v):
    return (np.asarray(v, np.float64).reshape(-1).view(np.uint64) >> np.uint64(32)).astype(np.uint32)


def test_high_words_order_as_the_test_needs():
    """outside() of ap_coarse.cuh: |dz|^2 at or above the radius (high words), every NaN and infinity above every
    radius, and nothing inside a radius of 0."""
    nan = np.uint64([0x7ff8000000000000, 0xfff8000000000000, 0x7fffffffffffffff, 0xffffffffffffffff]).view(np.float64)
    dz = np.concatenate([[0.0, 5e-324, 1e-300, 1e-8, 0.25, 1.0, 65536.0, 1e300, np.inf], nan])
    safe = np.array([0.0, 1e-300, 1e-8, 0.25, 16384.0])
    got = _high(dz)[:, None] >= _high(safe)[None]
    with np.errstate(invalid="ignore"):
        want = ~(dz[:, None] < safe[None])
    same_word = _high(dz)[:, None] == _high(safe)[None]
    assert np.array_equal(got, want | same_word)
    assert got[:, 0].all() and got[-5:].all()


@pytest.mark.gpu
@pytest.mark.parametrize("arith", [abi.AP_ARITH_REF_CPU, abi.AP_ARITH_REF_CUDA, abi.AP_ARITH_FAST])
@pytest.mark.parametrize("case", ["nan spacing", "infinite spacing", "overflowing coefficient"])
@pytest.mark.parametrize("ft", [0, 1, 4])
def test_not_a_number_ends_the_pixel(ft, case, arith):
    import torch

    import oracle
    if case == "overflowing coefficient" and ft != 4:
        pytest.skip("Multibrot only")
    n, W, H = 40, 13, 7
    z, orbit = 0j, []
    for _ in range(n + 1):  # z^n + z/4 - 0.1 + 0.1i stays bounded for all three formulas here
        orbit.append(z)
        z = (complex(abs(z.real), abs(z.imag)) ** 2 if ft == 1 else z ** 3 + 0.25 * z if ft == 4 else z * z) + (-0.1 + 0.1j)
    re, im = np.array([v.real for v in orbit]), np.array([v.imag for v in orbit])
    d = {"nan spacing": np.nan, "infinite spacing": np.inf}.get(case, 0.5)
    p = abi.new_params(width=W, height=H, max_iter=200, fractal_type=ft, tier=abi.AP_TIER_PERTURB, arith=arith, dx_hi=d,
                       dy_hi=d, ref_px=0.5 * (W - 1), ref_py=0.5 * (H - 1), ref_len=n, gen_n=3,
                       gen_kr=1.7e308 if d == 0.5 else 0.25, gen_ki=1.7e308 if d == 0.5 else 0.0,
                       flags=abi.AP_FLAG_REBASE | abi.AP_FLAG_NO_RGB)
    _, want_g, want_k = oracle.pert_grid(p, re, im, None, np.arange(W, dtype=np.float64), np.arange(H, dtype=np.float64))[:3]
    L = _lib.load()
    d_re, d_im = torch.from_numpy(re).cuda(), torch.from_numpy(im).cuda()
    po = torch.zeros((n + 1) * 6, dtype=torch.float64, device="cuda")
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(L.ap_pack_orbit(C.c_void_p(d_re.data_ptr()), C.c_void_p(d_im.data_ptr()), n, C.c_void_p(po.data_ptr()), st),
               "ap_pack_orbit")
    it = torch.empty((H, W), dtype=torch.float32, device="cuda")
    k = torch.empty((H, W), dtype=torch.int32, device="cuda")
    g = torch.empty((H, W), dtype=torch.uint8, device="cuda")
    b = abi.ApFrameBuffers()
    b.ref_re, b.ref_im, b.orbit_packed = (C.c_void_p(t.data_ptr()) for t in (d_re, d_im, po))
    b.iter_map, b.kmap, b.glitch_out = (C.c_void_p(t.data_ptr()) for t in (it, k, g))
    _lib.check(L.ap_render_pass(C.byref(p), C.byref(b), st), "ap_render_pass")
    assert np.array_equal(k.cpu().numpy(), want_k) and np.array_equal(g.cpu().numpy() != 0, want_g != 0)
    assert (want_k < 50).all()  # every pixel ends within one walk of the orbit
    assert want_g.any() or (case, arith) == ("overflowing coefficient", abi.AP_ARITH_FAST)  # there an infinity escapes
