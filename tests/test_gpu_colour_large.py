"""The kernels that large maps take (from 2^19 and 2^20 pixels on): the histogram counted in shared memory,
against the oracle's counts, and the colouring of four pixels a thread, bit for bit against the same
map coloured in strips below that size."""
import ctypes as C

import numpy as np
import pytest

import oracle
from fractura_b200 import _lib, abi

pytestmark = pytest.mark.gpu

# at the rule, one row of pixels below it, odd counts (the last pixels of a block of four), several
# shares of 65408 pixels a block
SHAPES = [(512, 1024), (511, 1024), (727, 723), (1081, 1919), (3100, 3203)]


def a_map(H, W, max_iter):
    rng = np.random.default_rng(H * 7919 + W)
    it = (rng.random((H, W)) * max_iter).astype(np.float32)
    it[: H // 3] = np.float32(3.25)                     # a flat stretch
    it[rng.random((H, W)) < 0.2] = -1.0
    it[-1, -5:] = [0.0, max_iter, 0.5, 2.0, -1.0]       # the ends of the bins
    it[H // 2] = -1.0
    return it


def on_device(it, offset):
    """The map on the device, `offset` floats past a 16-byte boundary."""
    import torch
    buf = torch.empty(it.size + 4, dtype=torch.float32, device="cuda")
    view = buf[offset:offset + it.size]
    view.copy_(torch.from_numpy(it.ravel()))
    return buf, view


@pytest.mark.parametrize("num_bins", [3, 2048, 65535, 65536, 65537])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("shape", SHAPES)
def test_histogram_of_a_large_map(shape, offset, num_bins):
    import torch
    H, W = shape
    max_iter = 700
    it = a_map(H, W, max_iter)
    keep, d_it = on_device(it, offset)
    hist = torch.full((num_bins,), 7, dtype=torch.int32, device="cuda")
    cdf = torch.zeros(num_bins, dtype=torch.float32, device="cuda")
    L = _lib.load()
    _lib.check(L.ap_histogram_cdf(C.c_void_p(d_it.data_ptr()), W, H, max_iter, num_bins,
                                  C.c_void_p(hist.data_ptr()), C.c_void_p(cdf.data_ptr()), None), "ap_histogram_cdf")
    fr = oracle.Frame(W, H)
    fr.iter_map[...] = it
    oracle.histogram_cdf(fr, max_iter, num_bins)
    assert np.array_equal(hist.cpu().numpy(), fr.hist)
    assert np.array_equal(cdf.cpu().numpy().view(np.uint32), fr.cdf.view(np.uint32))


def test_histogram_of_a_flat_map():
    """Every pixel in one bin: each block's counter reaches its share of the map."""
    import torch
    H, W = 3072, 4096
    hist = torch.zeros(65536, dtype=torch.int32, device="cuda")
    cdf = torch.zeros(65536, dtype=torch.float32, device="cuda")
    it = torch.full((H, W), 250.0, device="cuda")
    it[:, 17] = 251.0                                   # no warp of 128 pixels is flat
    L = _lib.load()
    _lib.check(L.ap_histogram_cdf(C.c_void_p(it.data_ptr()), W, H, 500, 65536, C.c_void_p(hist.data_ptr()),
                                  C.c_void_p(cdf.data_ptr()), None), "ap_histogram_cdf")
    got = hist.cpu().numpy()
    pos = [int((v * (1.0 / 500.0)) * 65535.0) for v in (250.0, 251.0)]
    assert got[pos[0]] == H * (W - 1) and got[pos[1]] == H and got.sum() == H * W


def coloured(it, rows, scheme, hdr, arith, lut, cdf, offset=0):
    import torch
    H, W = it.shape
    rgb = torch.full((H, W, 3), 9, dtype=torch.int16 if hdr else torch.uint8, device="cuda")
    keep, d_it = on_device(it, offset)
    L = _lib.load()
    for j in range(0, H, rows):
        p = abi.new_params(width=W, height=min(rows, H - j), factor=1, max_iter=700, scheme_id=scheme, num_bins=65536,
                           arith=arith, palette_offset=0.37, color_density=1.3, color_contrast=0.8, is_hdr=int(hdr))
        b = abi.ApFrameBuffers()
        b.iter_map = C.c_void_p(d_it[j * W:].data_ptr())
        b.rgb, b.lut = C.c_void_p(rgb[j:].data_ptr()), C.c_void_p(lut.data_ptr())
        if cdf is not None:
            b.cdf = C.c_void_p(cdf.data_ptr())
        _lib.check(L.ap_colour(C.byref(p), C.byref(b), None), "ap_colour")
    return rgb.cpu().numpy()


@pytest.mark.parametrize("hdr", [False, True])
@pytest.mark.parametrize("scheme", list(range(13)))
def test_colour_of_a_large_map_is_the_strips(scheme, hdr):
    import torch
    rng = np.random.default_rng(scheme)
    lut = torch.from_numpy((rng.random((2048, 3)) * (65535 if hdr else 255)).astype(np.float32)).cuda()
    cdf = torch.from_numpy(np.sort(rng.random(65536)).astype(np.float32)).cuda() if scheme == 11 else None
    for (H, W), offset in (((1024, 1024), 0), ((1031, 1028), 0), ((1031, 1028), 1)):
        it = a_map(H, W, 700)
        for arith in (abi.AP_ARITH_REF_CPU, abi.AP_ARITH_FAST):
            whole = coloured(it, H, scheme, hdr, arith, lut, cdf, offset)
            strips = coloured(it, 101, scheme, hdr, arith, lut, cdf)
            assert np.array_equal(whole, strips), (H, W, offset, arith)
