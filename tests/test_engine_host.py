"""The host side of single blocks (pa_engine.cu), compiled against a fake CUDA runtime (fake_runtime.cpp): what a call does
when one of the calls below it fails.  No GPU."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from privacyamplification_gb300 import FLAG_EXACT, DEFAULT_FLAGS

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "privacyamplification_gb300", "csrc")
PA_ERR_CUDA = -2


class Config(ctypes.Structure):
    _fields_ = [("device_id", ctypes.c_int32), ("max_sample_size", ctypes.c_uint32), ("reduction_exp", ctypes.c_uint32),
                ("pre_mul_reduction_exp", ctypes.c_uint32), ("residual_limit", ctypes.c_float)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("engine") / "engine.so"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    # -Bsymbolic: a CUDA runtime that the process has loaded must not take the fake one's place
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-w",
                        "-I", os.path.join(cuda, "include"), "-I", CSRC, "-x", "c++",
                        os.path.join(CSRC, "pa_engine.cu"), os.path.join(ROOT, "tests", "fake_runtime.cpp"),
                        "-o", str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = ctypes.CDLL(str(out))
    lib.fake_log.restype = ctypes.c_char_p
    lib.fake_held.restype = ctypes.c_size_t
    lib.fake_limit.argtypes = [ctypes.c_size_t]
    lib.fake_residual.argtypes = [ctypes.c_float]
    return lib


class Engine:
    def __init__(self, lib, n):
        self.lib, self.ptr = lib, ctypes.c_void_p()
        lib.fake_reset()
        self.rc = lib.pa_create(ctypes.byref(Config(0, n, 0, 0, 0.0)), ctypes.byref(self.ptr))

    def close(self):
        self.lib.pa_destroy(self.ptr)

    def set_seed(self, n, reuse=-1):
        return self.lib.pa_set_seed(self.ptr, words(n).ctypes.data_as(ctypes.c_void_p), n, reuse)

    def process(self, n, v, flags=DEFAULT_FLAGS):
        ks, kr, out = words(n), words(v), np.zeros(max(n // 16, v // 8), np.uint8)
        return self.lib.pa_process(self.ptr, *(a.ctypes.data_as(ctypes.c_void_p) for a in (ks, kr)), n, v, flags,
                                   out.ctypes.data_as(ctypes.c_void_p), None)


def words(bits):
    return np.zeros(bits // 32, np.uint32)


@pytest.mark.parametrize("n,flags,residual,fail,skip", [
    (1 << 16, DEFAULT_FLAGS, 0.0, "direct", 0),         # the block's own launch
    (1 << 16, DEFAULT_FLAGS, 0.0, "publish", 0),        # behind a short block
    (1 << 18, DEFAULT_FLAGS, 0.0, "key", 0),
    (1 << 18, DEFAULT_FLAGS, 0.0, "publish", 0),        # behind the FP32 passes
    (1 << 19, DEFAULT_FLAGS, 0.5, "exact_seed", 0),     # the guard's recompute
    (1 << 19, DEFAULT_FLAGS, 0.5, "exact", 0),
    (1 << 19, DEFAULT_FLAGS, 0.5, "publish", 1),        # behind the recompute
    (1 << 18, DEFAULT_FLAGS | FLAG_EXACT, 0.0, "publish", 0),
    (1 << 24, DEFAULT_FLAGS, 0.0, "copy_async", 1)])    # key_rest's copy, the key's being under way
def test_process_waits_before_it_returns_an_error(lib, n, flags, residual, fail, skip):
    """The caller's buffers, pinned ones above all, are not read after the call: whatever it queued has finished."""
    eng = Engine(lib, n)
    assert eng.rc == 0 and eng.set_seed(n) == 0
    lib.fake_reset()
    lib.fake_residual(residual)
    lib.fake_fail(fail.encode(), skip)
    assert eng.process(n, n // 4 + n // 8, flags) == PA_ERR_CUDA
    calls = lib.fake_log().decode().split("\n")[:-1]
    failed = [i for i, c in enumerate(calls) if c == fail][skip]
    assert "sync main" in calls[failed + 1:], calls
    if fail == "copy_async":
        assert "sync side" in calls[failed + 1:], calls
    lib.fake_reset()
    assert eng.process(n, n // 4 + n // 8, flags) == 0  # the engine goes on
    eng.close()


@pytest.mark.parametrize("h,v,flags,copies", [
    (393184, 512, DEFAULT_FLAGS, 0), (393216, 512, DEFAULT_FLAGS, 1),    # word by word: 48 KB, one word more
    (393216, 512, DEFAULT_FLAGS | FLAG_EXACT, 1), (1048576, 512, DEFAULT_FLAGS, 1),
    (655360, 393216, DEFAULT_FLAGS, 0), (655360, 393216, DEFAULT_FLAGS | FLAG_EXACT, 0),  # transforms: 80 KB
    (2097120, 1 << 20, DEFAULT_FLAGS, 0), (2097152, 1 << 20, DEFAULT_FLAGS, 1)])          # 256 KB, one word more
def test_pinned_keys_read_in_place(lib, h, v, flags, copies):
    """A pinned key that every cluster of CTAs reads again is copied above 48 KB, one that is read once above 256 KB."""
    eng = Engine(lib, h + v)
    assert eng.rc == 0 and eng.set_seed(h + v) == 0
    lib.fake_reset()
    assert eng.process(h + v, v, flags) == 0
    assert lib.fake_log().decode().split("\n").count("copy_async") == copies
    eng.close()


def test_set_seed_waits_before_it_returns_an_error(lib):
    eng = Engine(lib, 1 << 18)
    lib.fake_fail(b"seed", 0)
    assert eng.set_seed(1 << 18) == PA_ERR_CUDA
    calls = lib.fake_log().decode().split("\n")[:-1]
    assert "sync main" in calls[calls.index("seed") + 1:], calls
    eng.close()


BUFFER = 1 << 29  # 2^26 complex values


@pytest.mark.parametrize("logn,buffers", [(28, 7), (29, 13), (30, 25)])
def test_large_engine_fits_beside_other_tenants(lib, logn, buffers):
    """An engine above 2^27 bits needs what one chunk of 2^27 bits at a time takes (`buffers` with everything at the block's
    own length); more, where it can be had, holds transforms that are otherwise repeated."""
    n = 1 << logn
    eng = Engine(lib, n)
    assert eng.rc == 0
    most = lib.fake_held()
    eng.close()
    assert lib.fake_held() == 0
    small = 4 * (n // 8 + 256) + (1 << 24) + 256 + 304 * 65536 + 4096  # keys, seed, result, bit planes, park, words
    for limit in (most, most - 1, buffers * BUFFER + small):
        eng = Engine(lib, n)
        eng.close()
        lib.fake_limit(limit)
        eng.rc = lib.pa_create(ctypes.byref(Config(0, n, 0, 0, 0.0)), ctypes.byref(eng.ptr))
        assert eng.rc == 0 and lib.fake_held() <= limit, limit
        eng.close()
        assert lib.fake_held() == 0
    lib.fake_reset()
    lib.fake_limit(3 * BUFFER)  # not even the passes' own
    assert lib.pa_create(ctypes.byref(Config(0, n, 0, 0, 0.0)), ctypes.byref(eng.ptr)) == PA_ERR_CUDA
    assert lib.fake_held() == 0
    lib.fake_reset()
