"""The order of the samples of a supersampling pass (csrc/ap_samples.cuh, compiled for the host): every
place of every pixel once, and Python's integers where the number of a sample passes 32 bits."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fractura_b200", "csrc")


@pytest.fixture(scope="module")
def places(tmp_path_factory):
    d = tmp_path_factory.mktemp("samples")
    src = d / "samples.cpp"
    src.write_text('#include "ap_samples.cuh"\n'
                   'extern "C" void places(int f, int64_t n, const int64_t* q, int* out) {\n'
                   '    for (int64_t t = 0; t < n; ++t) ap::sample_place(q[t], f, out + 3 * t, out + 3 * t + 1, out + 3 * t + 2);\n'
                   '}\n')
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(d / "samples.so")], check=True)
    fn = C.CDLL(str(d / "samples.so")).places

    def call(f, q):
        q = np.ascontiguousarray(q, np.int64)
        out = np.empty((q.size, 3), np.int32)
        fn(C.c_int(f), C.c_int64(q.size), q.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
        return out
    return call


@pytest.mark.parametrize("f", [1, 2, 3, 4, 5, 8, 16])
def test_every_place_once_in_order(places, f):
    want = [(p, x, y) for p in range(32) for y in range(f) for x in range(f)]
    assert np.array_equal(places(f, np.arange(32 * f * f)), np.array(want))


@pytest.mark.parametrize("f", [8191, 8192, 23170, 23171, 46340, 46341, 65536, 2 ** 24])
def test_numbers_past_32_bits(places, f):
    total = 32 * f * f
    q = sorted({min(total - 1, max(0, v)) for c in (0, 2 ** 31, 2 ** 32, f * f, 4 * f * f, 31 * f * f, total) for v in range(c - 40, c + 40)})
    want = [(v // (f * f), v % (f * f) % f, v % (f * f) // f) for v in q]
    assert np.array_equal(places(f, q), np.array(want))
