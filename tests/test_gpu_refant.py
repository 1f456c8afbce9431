"""Reference-antenna pass of the mixed form (csrc/kernels_refant.cuh): its rows of avgData against the oracle where its
paths part: part of a 16-channel block, of a staged round (64 channels) and of a channel slab, more than 32 reference
baselines, directions that end inside a group of 8, and visibilities of very different sizes.

Tolerance relative to sum|V| of the row: the phasors of a block and of a channel offset are off by at most 3e-10 each
(float rounding of the angle 1.8e-10, of the correction 1.2e-10) and the second is held to sqrt(2) 2^-32 beside; the
rounding of v is at most 2^-8 2^-29 per component: 1e-9."""
import numpy as np
import pytest

import oracle
import leap_gb300 as lg
from leap_gb300 import synth

pytestmark = pytest.mark.gpu
TOL = 1e-9


def check(ctx, obs, dirs):
    md = lg.build_metadata(obs)
    ctx.set_metadata(md)
    ctx.set_integration(0, obs.vis, obs.uvw)
    dds = np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])
    ctx.calibrate(0, dds, lg.LEAP_PRECISION_MIXED)
    rows = np.asarray([i for i in md.I1 if i >= 0])
    mag = np.abs(obs.vis.astype(np.complex128)).reshape(obs.channels, obs.timesteps, obs.nbaselines, -1)[..., 0].sum(axis=(0, 1))
    for d in range(len(dirs)):
        exp = oracle.rotate_visibilities(obs.vis, obs.uvw, dds[d], obs.nbaselines, obs.freq_start_hz, obs.freq_inc_hz)
        err = np.abs(ctx.avgdata(d)[rows, 0] - exp[rows, 0])
        assert (err <= TOL * mag[rows]).all(), (d, (err / mag[rows]).max())


@pytest.mark.parametrize("stations,timesteps,channels", [(4, 1, 1), (9, 2, 15), (16, 3, 17), (34, 1, 64), (11, 2, 65),
                                                         (16, 1, 200), (40, 5, 48)])
@pytest.mark.parametrize("directions", [1, 7, 8, 9])
def test_reference_rows(ctx, stations, timesteps, channels, directions):
    check(ctx, *synth.small_case(stations=stations, timesteps=timesteps, channels=channels, directions=directions,
                                 vis_dtype=np.complex64, seed_shift=channels + directions))


@pytest.mark.parametrize("scale", [2.0 ** -90, 1.0, 2.0 ** 90])
def test_reference_rows_of_uneven_size(ctx, scale):
    """Rows of zeros, single samples 10^6 times the others, and all of it scaled."""
    obs, dirs = synth.small_case(stations=36, timesteps=2, channels=80, directions=3, vis_dtype=np.complex64)
    obs.vis[::23] *= 1e6
    obs.vis[::5] = 0
    obs.vis[:, ::7] = 0
    obs.vis *= np.float32(scale)
    check(ctx, obs, dirs)
