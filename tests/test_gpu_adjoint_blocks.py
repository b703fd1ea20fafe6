"""The derivative forward pass in blocks of untested steps with cycle detection: values, escape steps
and checkpoints (those of bounded pixels too) equal the pass at a checkpoint spacing of 7, which
leaves no room for a block, bit for bit; and the adjoint's gradient is the tangents' sum where pixels
are bounded, escape at once, or carry no gradient."""
import math

import numpy as np
import pytest

from fractura_b200 import adjoint as adj

pytestmark = pytest.mark.gpu
W, H = 61, 45
VIEWS = {
    "julia": ([0.0, 0.0, math.log(3.0), -0.12, 0.6], 2, 2),
    "mandelbrot": ([-0.3, 0.0, math.log(3.0), 0.0, 0.0], 0, 2),
    "multibrot3": ([0.0, 0.0, math.log(3.0), 0.1, 0.2], 4, 3),
    "multibrot5": ([0.1, 0.0, math.log(3.0), 0.1, 0.2], 4, 5),
    "large_parameter": ([0.0, 0.0, math.log(4.0), 200.0, 0.0], 4, 2),
}


def _used(max_iter, every, k):
    """Slots that hold a checkpoint of a pixel that escapes at step k (-1: never)."""
    last = max_iter - 1 if k < 0 else k
    return last // every + 1 if last >= 0 else 0


@pytest.mark.parametrize("max_iter", [1, 15, 16, 24, 25, 500, 2003])
@pytest.mark.parametrize("every", [16, 17, 112, 1024])
@pytest.mark.parametrize("name", sorted(VIEWS))
def test_blocks_equal_tested_steps(name, every, max_iter):
    th, ft, n = VIEWS[name]
    s0, k0, ck0 = (t.cpu().numpy() for t in adj.forward(th, W, H, max_iter, ft, n, ckpt_every=7))
    s1, k1, ck1 = (t.cpu().numpy() for t in adj.forward(th, W, H, max_iter, ft, n, ckpt_every=every))
    assert np.array_equal(k0, k1)
    assert np.array_equal(s0.view(np.uint64), s1.view(np.uint64))
    if every % 7 == 0:
        step = every // 7
        for (i, j), k in np.ndenumerate(k1):
            if k == -2:
                continue
            m = _used(max_iter, every, k)
            assert np.array_equal(ck1[i, j, :m].view(np.uint64), ck0[i, j, 0:m * step:step][:m].view(np.uint64)), (i, j, k)


@pytest.mark.parametrize("name", ["julia", "mandelbrot", "multibrot3", "multibrot5"])
def test_gradient_equals_the_tangents(name):
    """Per pixel: g times the forward-mode tangent, to 1e-9 of the pixel's largest term (both sum up to
    300 products of relative error 1e-15)."""
    import torch
    th, ft, n = VIEWS[name]
    s, k, ck = adj.forward(th, W, H, 300, ft, n)
    g = torch.randn((H, W), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    g[::3] = 0.0
    total, pix = adj.adjoint(th, g, k, ck, W, H, 300, ft, n, per_pixel=True)
    want = adj.forward_mode(th, W, H, 300, ft, n) * g[..., None]
    want[(k <= 0)] = 0.0
    scale = want.abs().amax(-1, keepdim=True)
    assert torch.all((pix - want).abs() <= 1e-9 * scale)
    assert torch.all(pix[::3] == 0.0) and torch.all(pix[k < 0] == 0.0)
    assert torch.allclose(total, pix.sum((0, 1)), rtol=1e-9, atol=float(pix.abs().sum()) * 1e-15)
