"""Device tables of the spectral window (update_spectrum of csrc/host_math.h) when an allocation or a copy fails: the call
returns the error, and the next one does not take the tables for uploaded."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "icrar-leap-accelerate_gb300", "csrc")
C_LIGHT = 299792458.0
WINDOWS = [(150e6, 40e3, 48), (150e6, 40e3, 96), (151e6, 40e3, 96), (151e6, 41e3, 20)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("spectrum") / "libspectrum.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", CSRC, "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "spectrum_check.cc"),
                    os.path.join(CSRC, "host_math.cc"), "-o", so], check=True)
    return ctypes.CDLL(so)


def call(lib, window, fail=0):
    f0, df, channels = window
    return lib.spectrum_call(ctypes.c_double(f0), ctypes.c_double(df), channels, fail)


def check(lib, window):
    f0, df, channels = window
    lam, inv, rho = np.zeros(channels), np.zeros(channels), np.zeros(channels, np.int32)
    assert lib.spectrum_read(channels, *(a.ctypes.data_as(ctypes.c_void_p) for a in (lam, inv, rho))) == 1
    exp = np.array([C_LIGHT / (f0 + float(c) * df) for c in range(channels)])
    np.testing.assert_array_equal(lam, exp)
    np.testing.assert_array_equal(inv, 1 / exp)
    return rho


@pytest.mark.parametrize("before", [None] + WINDOWS)
@pytest.mark.parametrize("window", WINDOWS)
@pytest.mark.parametrize("fail", [1, 2, 3, 4])
def test_a_failed_step_is_done_again(lib, before, window, fail):
    lib.spectrum_reset()
    if before:
        assert call(lib, before) == 0
        check(lib, before)
    rc = call(lib, window, fail)
    assert rc in (0, fail)
    assert rc == 0 or lib.spectrum_read(window[2], None, None, None) == 0
    # The same window, another one (with the first window's size), and the one before.
    for again in (window, WINDOWS[0], before or window):
        assert call(lib, again) == 0
        got = check(lib, again)
        lib.spectrum_reset()
        assert call(lib, again) == 0
        np.testing.assert_array_equal(got, check(lib, again))
        lib.spectrum_reset()
        if before:
            call(lib, before)
        call(lib, window, fail)


def test_nothing_is_done_for_the_same_window(lib):
    lib.spectrum_reset()
    assert call(lib, WINDOWS[1]) == 0
    for fail in (1, 2, 3, 4):
        assert call(lib, WINDOWS[1], fail) == 0
        check(lib, WINDOWS[1])
