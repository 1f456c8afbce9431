"""Split grid operand (grid_split_operand): gridded averages at channel counts around its 8-channel runs and
16-channel chunks, timestep and baseline counts around its 4 x 4 tiles, and pols and rows of very different size (a
power of two per baseline and pol).

Tolerance: the 3xFP16 product keeps 22 bits of each factor (2^-22 of the largest term of a tile, three of them
dropped or rounded: < 1e-6), the interpolation 1e-8, the sums 1e-7: the 2e-6 of sum|V| of the gridded kernel's own
tests.  The scale is that of a (baseline, pol, 4 timesteps) tile, so the bound is taken against sum max|V| there."""
import numpy as np
import pytest

import oracle
import leap_gb300 as lg
from leap_gb300 import synth
from leap_gb300._abi import LEAP_OPTION_GRIDDED_ROTATION

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stations,timesteps,channels", [(2, 1, 1), (5, 3, 8), (6, 4, 9), (7, 5, 15), (8, 2, 24), (9, 6, 31),
                                                         (4, 8, 33), (5, 1, 520)])
def test_operand_edges(ctx, stations, timesteps, channels):
    obs, dirs = synth.small_case(stations=stations, timesteps=timesteps, channels=channels, directions=5,
                                 vis_dtype=np.complex64, seed_shift=channels)
    obs.vis[..., 1] *= 2.0 ** 25
    obs.vis[..., 2] *= 2.0 ** -40
    obs.vis[:, 1::3] *= 2.0 ** 12
    obs.vis[:, 0, 3] = 0
    ctx.set_metadata(lg.build_metadata(obs))
    ctx.set_integration(0, obs.vis, obs.uvw)
    dds = np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])
    ctx.set_option(LEAP_OPTION_GRIDDED_ROTATION, 1)
    try:
        ctx.calibrate(0, dds, lg.LEAP_PRECISION_MIXED)
        got = [ctx.avgdata(d) for d in range(5)]
    finally:
        ctx.set_option(LEAP_OPTION_GRIDDED_ROTATION, 2)
    T, nbl = timesteps, obs.nbaselines
    mag = np.abs(obs.vis).reshape(channels, T, nbl, 4)
    tile = np.stack([mag[:, t0:t0 + 4].max(axis=(0, 1)) for t0 in range(0, T, 4)])
    bound = 2e-6 * sum(tile[t // 4] for t in range(T)) * channels
    for d in range(5):
        exp = oracle.rotate_visibilities(obs.vis, obs.uvw, dds[d], nbl, obs.freq_start_hz, obs.freq_inc_hz)
        assert (np.abs(got[d] - exp) <= bound).all()
