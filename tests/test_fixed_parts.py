"""Products in two parts (fx_part, fx_add_products of csrc/fixed_phase.h), on the CPU against whole numbers.

Tolerance, in units of 2^-56 of a full-scale product: a term rounds its cross products once (1/2) and drops two
products of remainders (1/4 each); a's and b's own rounding to 2^-33 of 2^-28 is 2^-5 units each."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "icrar-leap-accelerate_gb300", "csrc")
UNITS = 1 + 2 * 2.0 ** -5


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("parts") / "libparts.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(ROOT, "tests", "fixed_parts_check.cc"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.fx_parts_check.restype = ctypes.c_longlong
    return lib


def _sum(lib, a, b, x, y):
    keep = [np.ascontiguousarray(v, t) for v, t in ((a, np.float64), (b, np.float64), (x, np.int64), (y, np.int64))]
    return lib.fx_parts_check(len(a), *(v.ctypes.data_as(ctypes.c_void_p) for v in keep))


def _error(lib, a, b, x, y):
    # a x in units of 2^-56: a in 2^-28, x in 2^-60
    exact = sum(Fraction(float(p)) * int(q) / 2 ** 32 for p, q in zip(np.concatenate([a, b]), np.concatenate([x, y])))
    return abs(_sum(lib, a, b, x, y) - exact)


@pytest.mark.parametrize("n", [1, 2, 17, 64])
@pytest.mark.parametrize("scale", [1.0, 2.0 ** -20, 2.0 ** -40])
def test_sums(lib, n, scale):
    rng = np.random.default_rng(n)
    for _ in range(50):
        a, b = rng.uniform(-1, 1, (2, n)) * 2.0 ** 28 * scale
        t = rng.uniform(0, 2 * np.pi, n)
        x, y = (np.cos(t) * 2.0 ** 60).astype(np.int64), (np.sin(t) * 2.0 ** 60).astype(np.int64)
        assert _error(lib, a, b, x, y) <= n * UNITS


def test_extremes(lib):
    """Full-scale parts, remainders at either end, 64 equal terms (the most before the sums go to FP64), exact zeros."""
    top, one = 2.0 ** 28, 2 ** 60
    for a in (top, -top, np.nextafter(top, 0), top - 0.5, 0.5, -0.5, 2.0 ** -34, np.nextafter(0.5, 0), 12345.5):
        for x in (one, -one, one - 1, 2 ** 31, -(2 ** 31), 2 ** 31 - 1, 2 ** 32, -1, 0, 759250124994401280):
            for n in (1, 64):
                v, w = np.full(n, a), np.full(n, x, np.int64)
                assert _error(lib, v, np.zeros(n), w, w) <= n * UNITS
                half = np.full(n, x // 2, np.int64)
                assert _error(lib, v, -v, half, half) <= n * UNITS
    n = 64
    assert _sum(lib, np.zeros(n), np.zeros(n), np.full(n, one), np.full(n, -12345)) == 0
    assert _sum(lib, np.full(n, 7.25), np.full(n, -3.5), np.zeros(n), np.zeros(n)) == 0
