"""Grid windows (grid_windows in csrc/kernels_grid.cuh) where plain FP32 decides them and where the double-float path has
to: slopes of exactly zero, slopes within and far beyond half a turn, units with rows that end inside a quad.  A window
that missed a stencil would lose its terms.  Bar: that of the gridded kernel, 2e-6 of the sum of |terms|."""
import numpy as np
import pytest

import oracle
import leap_gb300 as lg
from leap_gb300 import synth
from test_gpu_gridded import AVG_TOL, _gridded, _scale

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stretch", [0.0, 1.0, 5.0, 30.0])
@pytest.mark.parametrize("stations,timesteps,channels,directions", [(6, 1, 16, 1), (11, 5, 40, 65)])
def test_windows(ctx, stretch, stations, timesteps, channels, directions):
    obs, dirs = synth.small_case(stations=stations, timesteps=timesteps, channels=channels, directions=directions,
                                 vis_dtype=np.complex64, seed_shift=int(stretch))
    uvw = np.ascontiguousarray(obs.uvw * stretch)
    ctx.set_metadata(lg.build_metadata(obs))
    ctx.set_integration(0, obs.vis, uvw)
    dds = np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])
    _gridded(ctx, lambda: ctx.calibrate(0, dds, lg.LEAP_PRECISION_MIXED))
    for d in range(directions):
        exp = oracle.rotate_visibilities(obs.vis, uvw, dds[d], obs.nbaselines, obs.freq_start_hz, obs.freq_inc_hz)
        assert (np.abs(ctx.avgdata(d) - exp) <= AVG_TOL * _scale(obs)).all(), d
    ctx.release_integration(0)
