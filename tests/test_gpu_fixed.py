"""All-FP64 rotate + average in fixed point (csrc/kernels_fixed.cuh): avgData against the oracle at the sizes
where the kernel branches: partial tiles, stages (16 channels), seeds (32), flushes (64 and 128), slab splits,
warps per block, pols and element types; and the rows that its integer sums leave out.

Tolerance.  The oracle adds N = timesteps * channels terms in FP64, so its own rounding is at most
N 2^-53 sum|V| per component; a term is off by its phasor, 2^-52 on either side, and an argument may be rounded
to its other neighbour (one unit in the last place, in one sample of 500).  Bound per average:
(N + 4) 2^-53 sum|V| + (2 + N / 500) ulp(largest argument) max|V|."""
import numpy as np
import pytest

import oracle
import leap_gb300 as lg
from leap_gb300 import synth

pytestmark = pytest.mark.gpu
C_LIGHT = 299792458.0


def _case(stations, timesteps, channels, pols, directions, dtype, seed=0, uvw_scale=1.0):
    obs, dirs = synth.small_case(stations=stations, timesteps=timesteps, channels=channels, pols=pols,
                                 directions=directions, vis_dtype=dtype, seed_shift=seed)
    obs.uvw = obs.uvw * uvw_scale
    return obs, np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])


def _check(ctx, obs, dds, lost=()):
    md = lg.build_metadata(obs)
    ctx.set_metadata(md)
    ctx.set_integration(0, obs.vis, obs.uvw)
    ctx.calibrate(0, dds, lg.LEAP_PRECISION_FP64)
    n, nbl = obs.timesteps * obs.channels, obs.nbaselines
    mag = np.abs(np.where(np.isnan(obs.vis).any(axis=2, keepdims=True), 0, obs.vis)).astype(np.float64)
    mag = mag.reshape(obs.channels, obs.timesteps, nbl, obs.pols)
    total, largest = mag.sum(axis=(0, 1)), mag.max(axis=(0, 1))
    nu = obs.freq_start_hz + max(0, obs.channels - 1) * obs.freq_inc_hz
    for d in range(len(dds)):
        with np.errstate(all="ignore"):
            exp = oracle.rotate_visibilities(obs.vis, obs.uvw, dds[d], nbl, obs.freq_start_hz, obs.freq_inc_hz)
            arg = 2 * np.pi * np.abs((obs.uvw @ dds[d][2]) - obs.uvw[:, 2]) * nu / C_LIGHT
            arg = np.nan_to_num(arg).reshape(obs.timesteps, nbl).max(axis=0)
            bound = (n + 4) * 2.0 ** -53 * total + ((2 + n / 500) * np.spacing(arg))[:, None] * largest
            got = ctx.avgdata(d)
            for b in lost:  # (the oracle skips every sample of such a row)
                assert np.isnan(got[b]).all()
                got[b] = exp[b] = 0
            for part in (np.real, np.imag):
                a, b = part(got), part(exp)
                np.testing.assert_array_equal(np.isnan(a), np.isnan(b))
                np.testing.assert_array_equal(np.isinf(a), np.isinf(b))
                np.testing.assert_array_equal(a[np.isinf(a)], b[np.isinf(b)])
                ok = np.isfinite(b)
                assert (np.abs(a - b)[ok] <= bound[ok]).all(), np.max(np.abs(a - b)[ok] / bound[ok])


@pytest.mark.parametrize("dtype,pols", [(np.complex64, 4), (np.complex64, 2), (np.complex64, 1), (np.complex128, 4),
                                        (np.complex128, 2), (np.complex128, 1)])
@pytest.mark.parametrize("stations,timesteps,channels,directions", [
    (2, 1, 1, 1), (7, 2, 15, 2), (8, 1, 16, 3), (9, 3, 17, 4), (8, 2, 32, 5), (8, 1, 33, 8), (7, 5, 63, 9), (16, 1, 65, 16),
    (5, 2, 128, 17), (5, 1, 129, 2), (6, 40, 20, 3), (4, 1, 300, 1)])
def test_shapes(ctx, dtype, pols, stations, timesteps, channels, directions):
    _check(ctx, *_case(stations, timesteps, channels, pols, directions, dtype, seed=channels + directions))


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_dynamic_range(ctx, dtype):
    """Pols, rows and channels of very different size, each within its own bound; denormals; zeros."""
    obs, dds = _case(8, 3, 70, 4, 5, dtype, seed=3)
    obs.vis[..., 1] *= 2.0 ** 30
    obs.vis[..., 2] *= 2.0 ** -60
    obs.vis[:, 5::9] *= 2.0 ** 40
    obs.vis[::7] *= 2.0 ** -20
    obs.vis[:, 11, 3] = 0
    obs.vis[:, 12, 3] = 1e-42
    _check(ctx, obs, dds)


@pytest.mark.parametrize("dtype,huge", [(np.complex64, 3e38), (np.complex128, 1.5e300)])
def test_rows_outside_the_exponent_range(ctx, dtype, huge):
    obs, dds = _case(8, 2, 40, 4, 3, dtype, seed=4)
    obs.vis[3, 5, 0] = np.inf
    obs.vis[4, 7, 2] = complex(0, -np.inf)
    obs.vis[5, 9, 1] = np.nan  # dropped with its group
    obs.vis[6, 11, 3] = huge
    obs.vis[:, 13] *= 1e-35 if dtype == np.complex64 else 1e-290
    _check(ctx, obs, dds)


@pytest.mark.parametrize("uvw_scale", [0.0, 1e-9, 30.0, 2000.0, 1e5])
def test_argument_range(ctx, uvw_scale):
    """Arguments from nothing to beyond 2^19 rad (where rows leave the integer sums), and a UVW that is not
    finite (its baseline is NaN, as the direct kernel makes it)."""
    obs, dds = _case(9, 2, 50, 4, 6, np.complex64, seed=5, uvw_scale=uvw_scale)
    _check(ctx, obs, dds)
    obs.uvw[3, 1] = np.nan
    obs.uvw[4, 0] = np.inf
    _check(ctx, obs, dds, lost=(3, 4))


@pytest.mark.parametrize("f0,df", [(120e6, -250e3), (12345.0, 98765.4), (1.4e9, 0.0), (-1e8, 1e6), (2e6, -1.1e5)])
def test_spectral_windows(ctx, f0, df):
    """Falling and wide bands; negative frequencies take the direct FP64 kernel."""
    obs, dds = _case(6, 1, 40, 4, 3, np.complex64, seed=6)
    obs.freq_start_hz, obs.freq_inc_hz = f0, df
    _check(ctx, obs, dds)
