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
                   'extern "C" int rows(int f) { return ap::sample_rows(f); }\n'
                   'extern "C" void places(int row0, int f, int64_t n, const int* q, int* out) {\n'
                   '    for (int64_t t = 0; t < n; ++t) ap::sample_place(row0, q[t], f, out + 3 * t, out + 3 * t + 1, out + 3 * t + 2);\n'
                   '}\n')
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(d / "samples.so")], check=True)
    lib = C.CDLL(str(d / "samples.so"))

    def call(row0, f, q):
        q = np.ascontiguousarray(q, np.int32)
        out = np.empty((q.size, 3), np.int32)
        lib.places(row0, f, C.c_int64(q.size), q.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p))
        return out
    return call, lib.rows


@pytest.mark.parametrize("f", [1, 2, 3, 4, 5, 8, 16])
def test_every_place_once_in_order(places, f):
    call, rows = places
    assert rows(f) >= 32 * f  # one part
    want = [(p, x, y) for p in range(32) for y in range(f) for x in range(f)]
    assert np.array_equal(call(0, f, np.arange(32 * f * f)), np.array(want))


@pytest.mark.parametrize("f", [5792, 5793, 8191, 8192, 23170, 23171, 46340, 46341, 65536, 2 ** 24])
def test_numbers_past_32_bits(places, f):
    """The ends of every part (the first and last hundred of them) against Python's integers."""
    call, rows = places
    step, total = rows(f), 32 * f
    assert step >= 1 and step * f <= 2 ** 30
    starts = list(range(0, total, step))
    for row0 in starts[:100] + starts[-100:]:
        n = min(step, total - row0) * f
        q = sorted({v for c in (0, f, n // 2, n) for v in range(max(0, c - 33), min(n, c + 33))})
        want = [((row0 * f + v) // (f * f), v % f, (row0 + v // f) % f) for v in q]
        assert np.array_equal(call(row0, f, q), np.array(want))
