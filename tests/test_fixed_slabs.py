"""Slab plans of the fixed-point kernels (choose_fixed_slabs of csrc/host_math.cc): every timestep and channel once,
and as many blocks as the GPU runs at a time wherever the call can be cut into so many, for any number of timesteps."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "icrar-leap-accelerate_gb300", "csrc")


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("slabs") / "libslabs.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "slabs_check.cc"), os.path.join(CSRC, "host_math.cc"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def call(timesteps, channels, base, resident):
        out = (ctypes.c_int * 4)()
        lib.slabs_check(timesteps, channels, ctypes.c_longlong(base), ctypes.c_longlong(resident), out)
        return tuple(out)
    return call


TIMESTEPS = [1, 2, 7, 14, 30, 31, 32, 33, 34, 40, 63, 64, 65, 100, 333, 400, 1000, 5000, 100000]


@pytest.mark.parametrize("channels", [1, 15, 16, 17, 48, 64, 129, 384, 1000])
@pytest.mark.parametrize("base", [1, 2, 5, 11, 21, 129, 258, 2064, 40000])
@pytest.mark.parametrize("resident", [456, 912, 1824])
def test_plans(plan, channels, base, resident):
    for timesteps in TIMESTEPS:
        t_per, c_per, nts, ncs = plan(timesteps, channels, base, resident)
        assert nts == -(-timesteps // t_per) and ncs == -(-channels // c_per)
        assert c_per % 16 == 0 or ncs == 1
        assert 1 <= nts * ncs <= 65535
        # Blocks of the finest cut: one timestep and one stage of 16 channels each.
        blocks, finest = base * nts * ncs, base * timesteps * -(-channels // 16)
        assert blocks >= min(finest, resident) / 2, (timesteps, t_per, c_per, nts, ncs)
        # Time in samples: rounds of blocks times a block's samples, against all of them spread evenly.
        length = -(-blocks // resident) * t_per * min(c_per, channels)
        even = base * timesteps * channels / resident
        if finest >= 64 * resident:
            assert length <= 2 * even
        if timesteps > 32:
            assert nts * ncs <= 32 or blocks <= 2 * resident


@pytest.mark.parametrize("channels", [48, 64, 384])
@pytest.mark.parametrize("base", [2, 5, 21])
def test_no_cliff(plan, channels, base):
    """One timestep more never makes the longest block of a round half as long again."""
    def time(t, resident=456):
        t_per, c_per, nts, ncs = plan(t, channels, base, resident)
        return -(-base * nts * ncs // resident) * t_per * min(c_per, channels)
    for t in range(1, 130):
        assert time(t + 1) <= max(1.5 * time(t), time(t) + channels)
