"""The periodic tail of a packed orbit (ap_pack_orbit's last record): the smallest period of the last
eight steps and the step it holds from, for periods, starts and lengths at the edges of the search and
of the blocks that compare the orbit, and none where there is none."""
import ctypes as C

import numpy as np
import pytest

from fractura_b200 import _lib

pytestmark = pytest.mark.gpu


def _tail(re, im):
    """-(4096 s0 + p) by the definition; 0 without a tail."""
    n = re.size
    last = n - 2
    if last < 128 or not re[-1] ** 2 + im[-1] ** 2 <= 65536.0:
        return 0.0
    for p in range(1, 4096):
        if 2 * p >= last:
            break
        j = last - np.arange(8)
        if np.all((re[j] == re[j - p]) & (im[j] == im[j - p])):
            k = np.arange(p, last + 1)
            bad = k[~((re[k] == re[k - p]) & (im[k] == im[k - p]))]
            s0 = bad[-1] + 1 - p if bad.size else 0
            return -(4096.0 * s0 + p)
    return 0.0


def _packed(re, im):
    import torch
    n = re.size
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (re, im)]
    out = torch.full((4 * n,), 7.0, dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().ap_pack_orbit(C.c_void_p(d[0].data_ptr()), C.c_void_p(d[1].data_ptr()), n - 1, C.c_void_p(out.data_ptr()),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)), "ap_pack_orbit")
    return out.cpu().numpy().reshape(n, 4)


@pytest.mark.parametrize("p,s0,n", [(1, 0, 130), (1, 60, 130), (1, 100, 400), (2, 17, 131), (3, 0, 2049), (64, 1000, 2305), (255, 7, 4097),
                                    (256, 300, 5000), (257, 2100, 9000), (4095, 0, 8193), (4095, 1, 8194), (4095, 2000, 20001),
                                    (4096, 0, 20000), (12, 5000, 16383), (12, 5000, 16384), (12, 250000, 303105), (12, 303000, 303105)])
def test_tail_is_found(p, s0, n):
    rng = np.random.default_rng(p + s0 + n)
    re, im = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    k = np.arange(s0 + p, n)
    re[k], im[k] = re[s0 + (k - s0) % p], im[s0 + (k - s0) % p]
    rec = _packed(re, im)
    assert rec[-1, 3] == _tail(re, im)
    assert np.array_equal(rec[:, 0], re) and np.array_equal(rec[:, 1], im) and rec[-1, 2] == 0.0
    re[n // 2] += 0.25  # one value of the tail off
    assert _packed(re, im)[-1, 3] == _tail(re, im)


def test_no_tail():
    rng = np.random.default_rng(3)
    re, im = rng.uniform(-1, 1, 5000), rng.uniform(-1, 1, 5000)
    assert _packed(re, im)[-1, 3] == 0.0
    re[:], im[:] = 0.5, 0.25
    assert _packed(re, im)[-1, 3] == -1.0
    for end in (300.0, np.inf, np.nan):  # escaped
        re[-1] = end
        assert _packed(re, im)[-1, 3] == 0.0
    assert _packed(re[:129], im[:129])[-1, 3] == 0.0  # too short
