"""Rows of complex<double> visibilities, and gradients of averages, down to the smallest subnormal numbers: the integer
sums leave them out, and the FP64 ones keep them.

Tolerance: sums of subnormal terms are rounded to 2^-1074 each: one unit for each product, in either form."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
import leap_gb300 as lg
from leap_gb300 import _abi, synth

pytestmark = pytest.mark.gpu
UNIT = 2.0 ** -1074


@pytest.mark.parametrize("scale", [2.0 ** -1030, 2.0 ** -1045, 2.0 ** -1060])
def test_averages(ctx, scale):
    obs, dirs = synth.small_case(stations=6, timesteps=2, channels=20, directions=3, vis_dtype=np.complex128)
    obs.vis[:, 3:9] *= scale
    ctx.set_metadata(lg.build_metadata(obs))
    ctx.set_integration(0, obs.vis, obs.uvw)
    dds = np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])
    ctx.calibrate(0, dds, lg.LEAP_PRECISION_FP64)
    rows = np.arange(3, 9)  # (their later timestep keeps its size: one timestep only is looked at below)
    ctx.set_integration(0, np.ascontiguousarray(obs.vis[:, :obs.nbaselines]), obs.uvw[:obs.nbaselines])
    ctx.calibrate(0, dds, lg.LEAP_PRECISION_FP64)
    for d in range(len(dds)):
        got = ctx.avgdata(d)[rows]
        exp = oracle.rotate_visibilities(np.ascontiguousarray(obs.vis[:, :obs.nbaselines]), obs.uvw[:obs.nbaselines], dds[d],
                                         obs.nbaselines, obs.freq_start_hz, obs.freq_inc_hz)[rows]
        assert np.abs(exp).max() > 100 * UNIT
        tol = 4 * obs.channels * UNIT + 1e-12 * np.abs(obs.vis[:, rows]).sum(axis=0)
        assert (np.abs((got - exp).real) <= tol).all() and (np.abs((got - exp).imag) <= tol).all()


@pytest.mark.parametrize("scale", [2.0 ** -1030, 2.0 ** -1055])
def test_gradients(ctx, scale):
    """dL/dV is linear in dL/dcal: that of a tiny one against that of one of ordinary size."""
    obs, dirs = synth.small_case(stations=5, timesteps=1, channels=9, directions=2, vis_dtype=np.complex128)
    ctx.set_metadata(lg.build_metadata(obs))
    ctx.set_integration(0, obs.vis, obs.uvw)
    dd = torch.from_numpy(np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs]).reshape(-1)).cuda()
    avg = torch.randn((2, obs.nbaselines), dtype=torch.complex128, generator=torch.Generator().manual_seed(1)).cuda()
    g = torch.randn((2, 5), dtype=torch.float64, generator=torch.Generator().manual_seed(2)).cuda()
    vis = torch.from_numpy(obs.vis).cuda()
    out = []
    for s in (1.0, scale):
        gs, gvis = g * s, torch.zeros_like(vis)
        lmn = torch.zeros((2, 3), dtype=torch.float64, device="cuda")
        ctx._check(_abi.lib.leap_backward(ctx.handle, 0, dd.data_ptr(), 2, avg.data_ptr(), gs.data_ptr(), vis.data_ptr(),
                                          lmn.data_ptr(), gvis.data_ptr(), ctypes.c_void_p(1)))
        torch.cuda.synchronize()
        out.append(gvis.cpu().numpy()[:, :, 0])
    exp = out[0] * scale
    assert np.abs(exp).max() > 100 * UNIT
    # Two sums over 5 stations, a quotient by |average|^2 and two products, each rounded to a unit: amplified by 1 / |average|.
    tol = 100 * UNIT / np.abs(avg.cpu().numpy()).min() + 1e-12 * np.abs(exp)
    assert (np.abs(out[1] - exp) <= tol).all()
