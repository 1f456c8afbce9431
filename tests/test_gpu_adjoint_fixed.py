"""Fixed-point adjoint kernels against the FP64 ones (which visibilities that are not 16-byte aligned still take):
dL/d(l, m, n) and dL/dV at the sizes where they branch (partial tiles, stages, seeds and flushes of channels, warps
per block, directions past 64, pols, element types), with NaN groups and rows that the integer sums leave out.

Tolerance: either form's phasors are good to 2^-49 and its sums to N 2^-53 of sum|terms|; the lmn sums have
N = rows * channels terms of |g| |V| 2 pi / lambda |uvw|, dL/dV has N = directions of |g|, then its own rounding
(2^-24 or 2^-53 of the result).  An argument that is rounded to its other neighbour in one form only adds 2^-52
of the argument (below 2^12 rad here): 2^-40 in all."""
import ctypes

import numpy as np
import pytest
import torch

import leap_gb300 as lg
from leap_gb300 import _abi, synth

pytestmark = pytest.mark.gpu
C_LIGHT = 299792458.0


def _offset_copy(x, dtype):
    """x's elements in memory that starts one 8-byte word past a 16-byte boundary."""
    flat = torch.zeros(x.numel() * x.element_size() // 8 + 2, dtype=torch.float64, device="cuda")
    v = flat[1:1 + x.numel() * x.element_size() // 8]
    v.copy_(torch.view_as_real(x).reshape(-1).view(torch.float64))
    return v


def _backward(ctx, dds, avg0, g_cal, vis_ptr, gvis_ptr):
    D = dds.shape[0]
    dd = torch.from_numpy(dds.reshape(-1)).cuda()
    g_lmn = torch.zeros((D, 3), dtype=torch.float64, device="cuda")
    ctx._check(_abi.lib.leap_backward(ctx.handle, 0, dd.data_ptr(), D, avg0.data_ptr(), g_cal.data_ptr(), vis_ptr,
                                      g_lmn.data_ptr(), gvis_ptr, ctypes.c_void_p(1)))
    torch.cuda.synchronize()
    return g_lmn.cpu().numpy()


def _case(ctx, stations, timesteps, channels, pols, directions, dtype, edit=None, seed=0):
    obs, dirs = synth.small_case(stations=stations, timesteps=timesteps, channels=channels, pols=pols, directions=directions,
                                 vis_dtype=dtype, seed_shift=seed)
    if edit:
        edit(obs)
    ctx.set_metadata(lg.build_metadata(obs))
    ctx.set_integration(0, obs.vis, obs.uvw)
    dds = np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])
    rng = np.random.default_rng(seed + 1)
    avg0 = torch.from_numpy(rng.standard_normal((directions, obs.nbaselines)) + 1j * rng.standard_normal((directions, obs.nbaselines))).cuda()
    g_cal = torch.from_numpy(rng.standard_normal((directions, stations))).cuda()
    vis = torch.from_numpy(obs.vis).cuda()
    gvis = torch.full_like(vis, 7)
    lmn = _backward(ctx, dds, avg0, g_cal, vis.data_ptr(), gvis.data_ptr())
    if pols == 1 and dtype == np.complex64:
        return  # 8-byte pieces: always the fixed-point form
    off, goff = _offset_copy(vis, dtype), _offset_copy(vis, dtype)
    exp = _backward(ctx, dds, avg0, g_cal, off.data_ptr(), goff.data_ptr())
    egvis = torch.view_as_complex(goff.view(torch.float32 if dtype == np.complex64 else torch.float64).reshape(-1, 2)).reshape(vis.shape)
    # scales of the sums: gradients of the averages are at most the largest |dL/dV|
    g = np.abs(egvis.cpu().numpy()).max()
    mag = np.abs(np.nan_to_num(obs.vis)).sum(axis=(0, 2)) * np.abs(np.nan_to_num(obs.uvw)).max(axis=1)
    scale = 2 * np.pi * (obs.freq_start_hz + channels * obs.freq_inc_hz) / C_LIGHT * g * mag.sum()
    n = obs.rows * channels
    np.testing.assert_array_equal(np.isfinite(lmn), np.isfinite(exp))
    ok = np.isfinite(exp)
    assert (np.abs(lmn - exp)[ok] <= (2.0 ** -40 + n * 2.0 ** -52) * scale).all()
    a, b = gvis.cpu().numpy(), egvis.cpu().numpy()
    out = 2.0 ** -23 if dtype == np.complex64 else 2.0 ** -52
    assert (np.abs(a - b) <= (2.0 ** -40 + directions * 2.0 ** -52) * directions * g + out * np.abs(b)).all()


@pytest.mark.parametrize("dtype,pols", [(np.complex64, 4), (np.complex64, 2), (np.complex64, 1)])
@pytest.mark.parametrize("stations,timesteps,channels,directions", [
    (3, 1, 1, 1), (7, 2, 15, 2), (8, 1, 16, 3), (9, 3, 17, 5), (8, 2, 33, 9), (12, 1, 130, 17), (6, 4, 20, 70)])
def test_shapes(ctx, dtype, pols, stations, timesteps, channels, directions):
    _case(ctx, stations, timesteps, channels, pols, directions, dtype, seed=channels)


def test_dropped_and_unusual_rows(ctx):
    def edit(obs):
        obs.vis[3, 5, 1] = np.nan
        obs.vis[4, 6, 0] = complex(0, np.nan)
        obs.vis[5, 7] *= 2.0 ** 40
        obs.vis[:, 8] = 0
        obs.vis[:, 9] *= 1e-36
        obs.uvw[10] *= 1e5  # beyond 2^19 rad
    _case(ctx, 8, 2, 40, 4, 6, np.complex64, edit, seed=3)
