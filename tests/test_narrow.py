"""Double to float on the integer pipe (csrc/narrow.h), bit for bit against the language's conversion."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "icrar-leap-accelerate_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("narrow") / "libnarrow.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(ROOT, "tests", "narrow_check.cc"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.narrow_check.restype = ctypes.c_longlong
    return lib


def check(lib, x):
    x = np.ascontiguousarray(np.concatenate([x, -x]))
    covered = ctypes.c_longlong()
    wrong = lib.narrow_check(x.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(x.size), ctypes.byref(covered))
    assert wrong == 0
    return covered.value


@pytest.mark.parametrize("exponent", [-126, -125, -1, 0, 1, 52, 126, 127])
def test_range_and_ties(lib, exponent):
    ulp = 2.0 ** -23
    m = np.array([1.0, 1 + ulp, 1 + 2 * ulp, 1.5, 2 - ulp])[:, None] + ulp * np.array([0, 0.5, 0.5 - 2.0 ** -29, 0.5 + 2.0 ** -29, 0.75])
    x = np.ldexp(np.minimum(m.ravel(), 2 - 2.0 ** -52), exponent)
    assert check(lib, x) == 2 * x.size


def test_random_and_uncovered(lib):
    rng = np.random.default_rng(3)
    x = np.frombuffer(rng.bytes(8 * 400000), np.float64)
    check(lib, x)
    assert check(lib, rng.standard_normal(100000)) == 200000
    assert check(lib, np.zeros(1)) == 2
    assert check(lib, np.array([5e-324, 2.0 ** -126 * (1 - 2.0 ** -53), 1e-45, 1e-310, 2.0 ** 128, 1e300, np.inf, np.nan])) == 0
