"""Pipelined mixed-precision kernel (csrc/kernels_pipe.cuh): avgData against the oracle where its paths part: 4, 2
or 1 tiles per block (up to 8, 16 and 32 directions), a warp with half of its directions, chunks of fewer than 16
channels, folds (64 channels), baselines that end inside a tile and tile groups that end inside a block.

Tolerance relative to sum|V| of the average: the step's phasor is off by 1.2e-7, hence w^k by at most
8 * 1.2e-7, z by 1e-7; Horner's rule rounds twice per channel, 2^-24 of a partial sum of at most 16 terms; the
64-channel sums round 4 times more: 1e-6 + 1e-7 + 32 * 2^-24 + 4 * 2^-24 < 3.3e-6."""
import numpy as np
import pytest

import oracle
import leap_gb300 as lg
from leap_gb300 import synth

pytestmark = pytest.mark.gpu
TOL = 3.3e-6


@pytest.mark.parametrize("stations,timesteps,channels", [(4, 1, 1), (9, 2, 15), (16, 3, 16), (23, 1, 17), (11, 2, 64),
                                                         (16, 1, 100), (23, 5, 48)])
@pytest.mark.parametrize("directions", [1, 3, 8, 9, 10, 12, 13, 16, 17, 27])
def test_pipelined_averages(ctx, stations, timesteps, channels, directions):
    obs, dirs = synth.small_case(stations=stations, timesteps=timesteps, channels=channels, directions=directions,
                                 vis_dtype=np.complex64, seed_shift=channels + directions)
    md = lg.build_metadata(obs)
    ctx.set_metadata(md)
    ctx.set_integration(0, obs.vis, obs.uvw)
    dds = np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])
    ctx.calibrate(0, dds, lg.LEAP_PRECISION_MIXED)
    mag = np.abs(obs.vis).reshape(channels, timesteps, obs.nbaselines, 4).sum(axis=(0, 1))
    for d in range(directions):
        exp = oracle.rotate_visibilities(obs.vis, obs.uvw, dds[d], obs.nbaselines, obs.freq_start_hz, obs.freq_inc_hz)
        err = np.abs(ctx.avgdata(d) - exp)
        assert (err <= TOL * np.sqrt(2) * mag).all(), (d, (err / mag).max())
