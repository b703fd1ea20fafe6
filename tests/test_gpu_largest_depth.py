"""The largest depth an int holds: pixels that settle on a cycle end there as bounded, in direct
iteration, in the second stage of perturbation and in the derivatives' forward pass -- block ends are
counted back from the depth, not past it."""
import ctypes as C

import numpy as np
import pytest

from fractura_b200 import _lib, abi
from fractura_b200 import adjoint as adj

pytestmark = pytest.mark.gpu
DEPTH = 2 ** 31 - 1
W, H = 17, 9


def _render(p, **buffers):
    import torch
    it = torch.empty((H, W), dtype=torch.float32, device="cuda")
    k = torch.full((H, W), -7, dtype=torch.int32, device="cuda")
    b = abi.ApFrameBuffers()
    b.iter_map, b.kmap = C.c_void_p(it.data_ptr()), C.c_void_p(k.data_ptr())
    for name, t in buffers.items():
        setattr(b, name, C.c_void_p(t.data_ptr()))
    _lib.check(_lib.load().ap_render_pass(C.byref(p), C.byref(b), C.c_void_p(torch.cuda.current_stream().cuda_stream)),
               "ap_render_pass")
    return k.cpu().numpy()


def _params(ft, **kw):
    return abi.new_params(width=W, height=H, factor=1, max_iter=DEPTH, fractal_type=ft, mode=abi.AP_MODE_COARSE,
                          flags=abi.AP_FLAG_NO_RGB, julia_cx_hi=-0.1, julia_cy_hi=0.1, gen_n=3, gen_kr=0.1, gen_ki=0.1, **kw)


@pytest.mark.parametrize("arith", [abi.AP_ARITH_REF_CPU, abi.AP_ARITH_REF_CUDA])
@pytest.mark.parametrize("ft", [2, 4])  # attracting fixed points
def test_direct(ft, arith):
    k = _render(_params(ft, tier=abi.AP_TIER_FP64, arith=arith, x_min_hi=-0.1, y_max_hi=0.1, dx_hi=0.2 / (W - 1), dy_hi=0.2 / (H - 1)))
    assert (k == -1).all()


@pytest.mark.parametrize("ft", [0, 2, 4])
def test_second_stage(ft):
    import torch
    n, z, o = 20, 0j, []
    for _ in range(n + 1):
        o.append(z)
        z = (z ** 3 + (0.1 + 0.1j) * z if ft == 4 else z * z) + (-0.1 + 0.1j)
    re, im = (torch.tensor([getattr(v, part) for v in o], dtype=torch.float64, device="cuda") for part in ("real", "imag"))
    po = torch.zeros(6 * (n + 1), dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().ap_pack_orbit(C.c_void_p(re.data_ptr()), C.c_void_p(im.data_ptr()), n, C.c_void_p(po.data_ptr()),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)), "ap_pack_orbit")
    k = _render(_params(ft, tier=abi.AP_TIER_PERTURB, dx_hi=1e-3, dy_hi=1e-3, ref_px=8.0, ref_py=4.0, ref_len=n, ref_cx=-0.1,
                        ref_cy=0.1), ref_re=re, ref_im=im, orbit_packed=po)
    assert (k == -1).all()


@pytest.mark.parametrize("ft,n,c", [(2, 2, -0.1), (4, 3, 0.1)])
def test_derivatives_forward(ft, n, c):
    _, k, _ = adj.forward([0.0, 0.0, np.log(0.2), c, 0.1], W, H, DEPTH, ft, n, ckpt=False)
    assert (k.cpu().numpy() == -1).all()
