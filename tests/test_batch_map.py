"""The order in which the batch queue runs through a tile (csrc/ap_batch_map.cuh, compiled for the
host): a permutation of the tile's pixels, at the numbers of patches where it is not scattered and at
those whose groups of 32 pixels no longer fit 32 bits."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractura_b200", "csrc")


@pytest.fixture(scope="module")
def scatter(tmp_path_factory):
    d = tmp_path_factory.mktemp("map")
    src = d / "map.cpp"
    src.write_text('#include "ap_batch_map.cuh"\n'
                   'extern "C" void scatter(int64_t patches, int64_t n, const int64_t* u, int64_t* local, int* w) {\n'
                   '    for (int64_t t = 0; t < n; ++t) local[t] = ap::batch_scatter(patches, u[t] >> 8, (int)(u[t] & 255), w + t);\n'
                   '}\n')
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(d / "map.so")], check=True)
    f = C.CDLL(str(d / "map.so")).scatter

    def call(patches, u):
        u = np.ascontiguousarray(u, np.int64)
        local, w = np.empty(u.size, np.int64), np.empty(u.size, np.int32)
        f(C.c_int64(patches), C.c_int64(u.size), u.ctypes.data_as(C.c_void_p), local.ctypes.data_as(C.c_void_p),
          w.ctypes.data_as(C.c_void_p))
        return local, w
    return call


@pytest.mark.parametrize("patches", [1, 2, 3, 7, 64, 841, 7918, 7919, 7920, 15838])
def test_every_pixel_once(scatter, patches):
    local, w = scatter(patches, np.arange(patches * 256))
    assert np.array_equal(np.sort(local * 256 + w), np.arange(patches * 256))


@pytest.mark.parametrize("patches", [2 ** 28 + 1, 2 ** 29 - 1, 2 ** 29, 2 ** 29 + 1, 2 ** 30, 2 ** 31 - 1])
def test_patches_whose_groups_pass_32_bits(scatter, patches):
    """Against the same arithmetic in Python's integers, at both ends and in between."""
    rng = np.random.default_rng(patches)
    items = np.concatenate([[0, 1, patches - 1], rng.integers(0, patches, 500)])
    u = np.concatenate([items * 256 + q for q in (0, 31, 32, 255)])
    local, w = scatter(patches, u)
    groups = patches * 8
    for a, got, gw in zip(u.tolist(), local.tolist(), w.tolist()):
        g = a // 32 if patches % 7919 == 0 else a // 32 * 7919 % groups
        assert (got, gw) == (g // 8, g % 8 * 32 + a % 32) and 0 <= got < patches
    assert np.unique(local * 256 + w).size == np.unique(u).size
