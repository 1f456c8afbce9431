"""Fixed-point phasors of the all-FP64 form (csrc/fixed_phase.h), on the CPU against exp(i fl(sf / lambda_c))
in 80 significant digits, sf / lambda_c being the reference's rounded argument.

Tolerance, in units of 2^-60 per component.  A 60-bit complex product rounds by 1 and drops low products
of up to 1 from their mean: 2 units.  A seed is two products of operands that are rounded once each: 7.
A step multiplies by the channel step's phasor, itself such a product (7), turned with one more rounding
(1): 2 + 7 + 1 = 10 per step, so 7 + 31 * 10 = 317 at the end of a block of 32 channels, and 2^-56 is 16.
The argument is off by an LSB at most, 2^(E - 63) rad for arguments below 2^E: 2^(E - 3) units more.
An argument may be rounded to the other neighbour, one unit in its last place off, only where sf / lambda_c
is within 2^-14 LSB of the tie between the two (phase, correction and their product are each good to a few
2^-18 LSB)."""
import ctypes
import os
import subprocess

import mpmath
import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "icrar-leap-accelerate_gb300", "csrc")
C_LIGHT = 299792458.0
SEED_EVERY = 32
UNITS = 317.0


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fx") / "libfx.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-I", CSRC, "-I",
                    os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "fixed_phase_check.cc"),
                    os.path.join(CSRC, "host_math.cc"), "-o", so], check=True)
    return ctypes.CDLL(so)


def wavelengths(f0, df, channels):
    return np.array([C_LIGHT / (f0 + float(c) * df) for c in range(channels)])


def phasors(lib, sf, f0, df, channels, c0=0):
    lam = wavelengths(f0, df, channels)
    zr, zi = np.zeros(channels, np.int64), np.zeros(channels, np.int64)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    rc = lib.fx_check(ctypes.c_double(sf), ctypes.c_double(f0), ctypes.c_double(df), channels, p(lam), c0, SEED_EVERY,
                      p(zr), p(zi))
    return rc, lam, zr[:channels - c0], zi[:channels - c0]


@pytest.mark.parametrize("f0,df,channels", [(150e6, 40e3, 130), (100e6, 5.4e3, 70), (700e6, 1e6, 48), (1.5e9, -3.7e5, 65),
                                            (139195000.0, 0.0, 33), (12345.678, 9876.54321, 64), (1.23456789e8, 1 / 3, 40)])
@pytest.mark.parametrize("scale", [0.0, 1e-320, 1e-12, 1e-3, 0.7, 40.0, -235.0, 4321.0, -1.5e5, 1.9e5])
def test_phasors_follow_the_rounded_argument(lib, f0, df, channels, scale):
    rng = np.random.default_rng(int(abs(scale) * 1000) % 99991 + channels)
    mpmath.mp.prec = 270
    kmax = 1 / wavelengths(f0, df, channels).min()
    for c0 in (0, 5):
        sf = scale * (1 + 0.1 * rng.uniform()) / kmax if abs(scale) > 1e-300 else scale
        rc, lam, zr, zi = phasors(lib, sf, f0, df, channels, c0)
        assert rc == 0
        worst = 0.0
        lsb = mpmath.mpf(2) ** (max(4, int(mpmath.floor(mpmath.log(max(abs(sf) * kmax, 1e-300), 2))) + 1) - 63)
        for k, c in enumerate(range(c0, channels)):
            arg = sf / lam[c]
            z = mpmath.expj(mpmath.mpf(float(arg)))
            err = max(abs(mpmath.mpf(int(zr[k])) - z.real * 2 ** 60), abs(mpmath.mpf(int(zi[k])) - z.imag * 2 ** 60))
            ulp = float(np.spacing(abs(arg))) * 2.0 ** 60
            bound = UNITS + lsb * 2 ** 60
            if err > bound and err <= bound + ulp:
                quotient = mpmath.mpf(sf) / mpmath.mpf(float(lam[c]))
                tie = mpmath.mpf(float(arg)) + mpmath.sign(quotient - float(arg)) * mpmath.mpf(float(np.spacing(abs(arg)))) / 2
                assert abs(quotient - tie) <= lsb / 2 ** 14
                continue
            worst = max(worst, float(err / bound))
        assert worst <= 1.0, worst


def test_range_limits(lib):
    kmax = 1 / wavelengths(150e6, 40e3, 32).min()
    for sf in (2.0 ** 19 / kmax * 1.01, np.inf, -np.inf, np.nan, 1e300):
        assert phasors(lib, sf, 150e6, 40e3, 32)[0] == 1
    for f0, df in ((0.0, 40e3), (-1e8, 40e3), (1e6, -1e6), (np.inf, 1.0), (1e8, np.nan)):
        with np.errstate(all="ignore"):
            try:
                rc = phasors(lib, 1.0, f0, df, 4)[0]
            except ZeroDivisionError:
                continue
        assert rc == 1
