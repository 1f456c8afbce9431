"""leap_backward against its formula in extended precision (numpy longdouble: 64 or 113 bits), for each element type and
pol count, with dropped groups, and up to 1024 directions.

Tolerances, units of 2^-53.  A gradient of the averages takes three sums over at most S stations, in FP64: S + 8 of its
terms' sizes at most for each that enters (G below: the same chain on absolute values), which two sums double:
2 S + 8.  Phasors, splits and sums of products are good to 4, a rounding of the result to 1: 2 S + 16.  dL/dV's errors
of different directions are independent, so their rms is at most that of sqrt(sum_d G^2), and no element is off by more
than sum_d G.  dL/d(l, m, n) also adds up its rows in FP64: one unit of sum|terms| for each.  complex<float> results
are rounded to 2^-24."""
import ctypes

import numpy as np
import pytest
import torch

import leap_gb300 as lg
from leap_gb300 import _abi, synth

pytestmark = pytest.mark.gpu
C_LIGHT = 299792458.0
L = np.longdouble
EPS = 2.0 ** -53


def _dropped(vis):
    return (np.isnan(vis.real) | np.isnan(vis.imag)).any(axis=2)


def _chain(md, avg, g_cal):
    """dL/d(averages), and the same on absolute values."""
    nI = md.A.shape[0] - 1
    A, Ad, Ad1 = (np.asarray(m, dtype=L) for m in (md.A[:nI], md.Ad[:, :nI], md.Ad1[:, :len(md.I1)]))
    size = np.abs(avg)
    factor = 1j * avg / (avg.real ** 2 + avg.imag ** 2)
    out = []
    for A_, Ad_, Ad1_, g, sign in ((A, Ad, Ad1, g_cal.astype(L), -1), (abs(A), abs(Ad), abs(Ad1), abs(g_cal.astype(L)), 1)):
        dphi = g @ Ad_
        cal1 = g + sign * 2 * L(np.pi) * (dphi @ A_)
        phi1 = cal1 @ Ad1_
        real = np.zeros(avg.shape, dtype=L)
        real[:, :nI] = dphi
        for k, b in enumerate(md.I1):
            real[:, b] += phi1[:, k]
        out.append(real)
    return out[0] * factor, out[1] / size


def _case(ctx, stations, timesteps, channels, pols, directions, dtype, edit=None, seed=0, uvw_scale=1.0):
    obs, dirs = synth.small_case(stations=stations, timesteps=timesteps, channels=channels, pols=pols, directions=directions,
                                 vis_dtype=dtype, seed_shift=seed)
    if edit:
        edit(obs)
    obs.uvw = obs.uvw * uvw_scale
    md = lg.build_metadata(obs)
    ctx.set_metadata(md)
    ctx.set_integration(0, obs.vis, obs.uvw)
    dds = np.stack([lg.dd_matrix(*obs.phase_centre, r, d) for r, d in dirs])
    rng = np.random.default_rng(seed + 1)
    nbl, S = obs.nbaselines, stations
    avg = rng.uniform(0.5, 2, (directions, nbl)) * np.exp(1j * rng.uniform(-np.pi, np.pi, (directions, nbl)))
    g_cal = rng.standard_normal((directions, S))
    vis = torch.from_numpy(obs.vis).cuda()
    gvis = torch.full_like(vis, 7)
    dd, avg_d, g_d = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (dds.reshape(-1), avg, g_cal))
    g_lmn = torch.full((directions, 3), 7, dtype=torch.float64, device="cuda")
    ctx._check(_abi.lib.leap_backward(ctx.handle, 0, dd.data_ptr(), directions, avg_d.data_ptr(), g_d.data_ptr(),
                                      vis.data_ptr(), g_lmn.data_ptr(), gvis.data_ptr(), ctypes.c_void_p(1)))
    torch.cuda.synchronize()
    got_vis, got_lmn = gvis.cpu().numpy(), g_lmn.cpu().numpy()

    g_avg, G = _chain(md, avg.astype(np.clongdouble), g_cal)
    drop = _dropped(obs.vis)
    v0 = np.where(drop, 0, obs.vis[:, :, 0]).astype(np.clongdouble)
    lam = C_LIGHT / (obs.freq_start_hz + np.arange(channels) * obs.freq_inc_hz)
    row = np.arange(obs.rows) % nbl
    exp_vis = np.zeros((channels, obs.rows), dtype=np.clongdouble)
    var, total = np.zeros(obs.rows, dtype=L), np.zeros(obs.rows, dtype=L)
    unit = (2 * S + 16) * EPS
    for d in range(directions):
        u, v, w = obs.uvw.T
        sf = -2 * np.pi * ((dds[d][2, 0] * u + dds[d][2, 1] * v + dds[d][2, 2] * w) - w)
        arg = (sf[None, :] / lam[:, None]).astype(L)
        z = np.cos(arg) + 1j * np.sin(arg)
        g = g_avg[d, row]
        exp_vis += g[None, :] * np.conj(z)
        var += G[d, row] ** 2
        total += G[d, row]
        k = -2 * L(np.pi) / lam.astype(L)[:, None]
        lmn = ((np.conj(g)[None, :] * 1j * v0 * z).real * k) @ obs.uvw.astype(L)
        scale = (G[d, row][None, :] * np.abs(v0) * np.abs(k)) @ np.abs(obs.uvw.astype(L))
        assert (np.abs(got_lmn[d] - lmn.sum(axis=0)) <= (unit + obs.rows * EPS) * scale.sum(axis=0)).all(), d
    exp_vis[drop] = 0
    assert (got_vis[:, :, 1:] == 0).all()
    assert (got_vis[:, :, 0][drop] == 0).all()
    err = np.abs(got_vis[:, :, 0] - exp_vis)
    out = 2.0 ** -24 if dtype == np.complex64 else 0
    assert (err <= unit * total[None, :] + out * np.abs(exp_vis)).all()
    if dtype == np.complex128:
        rms, bound = np.sqrt((err ** 2).mean()), np.sqrt(var.mean())
        assert rms <= unit * bound, rms / (EPS * bound)
    return err / EPS, exp_vis


@pytest.mark.parametrize("dtype,pols", [(np.complex64, 1), (np.complex64, 4), (np.complex128, 1), (np.complex128, 2),
                                        (np.complex128, 4)])
@pytest.mark.parametrize("stations,timesteps,channels,directions", [
    (3, 1, 1, 1), (7, 2, 15, 2), (8, 1, 16, 3), (9, 3, 17, 5), (8, 2, 33, 9), (12, 1, 130, 17), (6, 4, 20, 64), (6, 2, 20, 65),
    (5, 1, 9, 129)])
def test_shapes(ctx, dtype, pols, stations, timesteps, channels, directions):
    _case(ctx, stations, timesteps, channels, pols, directions, dtype, seed=channels)


@pytest.mark.parametrize("uvw_scale", [0.0, 0.001, 1.0, 20.0])
@pytest.mark.parametrize("directions", [256, 1024])
def test_many_directions(ctx, directions, uvw_scale):
    _case(ctx, 5, 1, 20, 1, directions, np.complex128, seed=7, uvw_scale=uvw_scale)


@pytest.mark.parametrize("dtype,pols", [(np.complex64, 1), (np.complex64, 2), (np.complex64, 4), (np.complex128, 1),
                                        (np.complex128, 2), (np.complex128, 4)])
def test_dropped_groups_and_unusual_rows(ctx, dtype, pols):
    def edit(obs):
        obs.vis[3, 5, -1] = np.nan
        obs.vis[4, 6, 0] = complex(0, np.nan)
        obs.vis[5, 7] *= 2.0 ** 40
        obs.vis[:, 8] = 0
        obs.vis[:, 9] *= 1e-36
    _case(ctx, 8, 2, 40, pols, 6, dtype, edit, seed=3)
