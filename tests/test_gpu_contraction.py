"""The FP64 contractions with Ad where their tiles and groups of directions end: cal phases against the oracle, and
gradients of several directions (summed over the lanes 16 at a time) against those of one direction each (one by one).

Tolerance of the gradients: the two sums over S stations differ by S 2^-52 of their terms, what follows by 2^-40 of its
scale (fixed-point sums): 2^-38 of the largest entry times sqrt(terms) is above both."""
import ctypes

import numpy as np
import pytest
import torch

import leap_gb300 as lg
from leap_gb300 import _abi, synth
from test_gpu_parity import FP64_CAL_TOL, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stations", [5, 24, 66])
@pytest.mark.parametrize("directions", [1, 3, 4, 13, 16, 17, 33])
def test_cal_phases(ctx, stations, directions):
    obs, dirs = synth.small_case(stations=stations, timesteps=1, channels=3, directions=directions, vis_dtype=np.complex64)
    md, mdo, dds, cal, cal_o, avg_o = run_case(ctx, obs, dirs, lg.LEAP_PRECISION_FP64)
    assert np.abs(cal - cal_o).max() <= FP64_CAL_TOL


@pytest.mark.parametrize("stations", [7, 40])
@pytest.mark.parametrize("directions", [4, 16, 17, 35])
def test_gradients_of_several_directions(ctx, stations, directions):
    obs, dirs = synth.small_case(stations=stations, timesteps=1, channels=4, directions=directions, vis_dtype=np.complex128)
    ctx.set_metadata(lg.build_metadata(obs))
    ctx.set_integration(0, obs.vis, obs.uvw)
    dds = np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])
    rng = np.random.default_rng(directions)
    avg0 = torch.from_numpy(rng.standard_normal((directions, obs.nbaselines)) + 1j * rng.standard_normal((directions, obs.nbaselines))).cuda()
    g_cal = torch.from_numpy(rng.standard_normal((directions, stations))).cuda()
    vis = torch.from_numpy(obs.vis).cuda()

    def backward(sel):
        dd = torch.from_numpy(dds[sel].reshape(-1)).cuda()
        n = len(sel)
        a, g = avg0[sel].contiguous(), g_cal[sel].contiguous()
        lmn = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
        gvis = torch.zeros_like(vis)
        ctx._check(_abi.lib.leap_backward(ctx.handle, 0, dd.data_ptr(), n, a.data_ptr(), g.data_ptr(), vis.data_ptr(),
                                          lmn.data_ptr(), gvis.data_ptr(), ctypes.c_void_p(1)))
        torch.cuda.synchronize()
        return lmn.cpu().numpy(), gvis.cpu().numpy()

    lmn, gvis = backward(list(range(directions)))
    one = [backward([d]) for d in range(directions)]
    tol = 2.0 ** -38
    exp = np.concatenate([o[0] for o in one])
    assert (np.abs(lmn - exp) <= tol * np.sqrt(obs.rows * 4) * np.abs(exp).max()).all()
    exp = sum(o[1] for o in one)
    assert (np.abs(gvis - exp) <= tol * np.sqrt(directions) * np.abs(exp).max()).all()
