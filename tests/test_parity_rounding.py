"""The parity rounding of the FP32 passes' last step (pa_parity.cuh), compiled for the host, over both signs around the
powers of two where FP32's spacing changes: the nearest integer's parity and the distance to it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = """
#include "pa_parity.cuh"
extern "C" void parity(const float* v, float* p, long n) { for (long i = 0; i < n; ++i) p[i] = pa::parity_half(v[i]); }
"""


@pytest.fixture(scope="module")
def parity(tmp_path_factory):
    d = tmp_path_factory.mktemp("parity")
    src, lib = d / "parity.cpp", d / "parity.so"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-I", os.path.join(ROOT, "privacyamplification_gb300", "csrc"),
                    str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(str(lib)).parity

    def run(v):
        v = np.ascontiguousarray(v, np.float32)
        p = np.empty_like(v)
        fn(v.ctypes.data_as(ctypes.c_void_p), p.ctypes.data_as(ctypes.c_void_p), ctypes.c_long(v.size))
        return p > 0, np.abs(np.abs(p) - np.float32(0.5))
    return run


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("power", [0, 4, 12, 21, 22, 23, 24])
def test_whole_numbers(parity, sign, power):
    ints = np.arange(max(0, (1 << power) - 5000), min((1 << power) + 5000, 1 << 24))
    odd, distance = parity((sign * ints).astype(np.float32))
    assert np.array_equal(odd, ints % 2 == 1)
    assert not distance.any()


@pytest.mark.parametrize("magnitude", [1.0, 1e3, 1e5, 4e6])
def test_fractions(parity, magnitude):
    v = np.random.default_rng(int(magnitude)).uniform(-magnitude, magnitude, 200000).astype(np.float32)
    near = np.rint(v.astype(np.float64))
    odd, distance = parity(v)
    want = np.abs(v - near)
    tie = want == 0.5  # of either parity
    assert np.array_equal(odd[~tie], near[~tie] % 2 != 0)
    assert np.abs(distance - want).max() <= 2.0 ** -26  # d - 1/2 is rounded once, below 1/2 in magnitude
