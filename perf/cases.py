"""Timed cases: what a program that calibrates with this framework has it do.

Each case is a dict of plain values; ``prepare`` makes the inputs and the handle that such a
program holds, ``run`` is one pass through the public entry points, ``exact`` the same result
from plain torch in 64 bits.  Four kinds of work:

resident  the integration is in a slot already and is calibrated towards a set of directions
          (``Context.calibrate``, or ``Context.calibrate_async`` from device tensors);
upload    a new integration goes into the slot, in MeasurementSet or Integration order, from
          host or device memory, and is calibrated: one solution interval of a run;
batched   ``Context.calibrate_batched`` over many integration chunks of uneven size;
grad      ``calibrate_lm``: cal phases and their gradients with respect to the directions and
          the visibilities.

``form`` is the library's arithmetic form.  The all-FP64 form's phases are returned as they come;
the mixed form's are good to the 1e-5 rad that it promises, and the programs that choose it hold
them in float32, beside the complex64 visibilities that they correct.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "icrar-leap-accelerate_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import leap_gb300 as lg  # noqa: E402
from leap_gb300 import synth  # noqa: E402
from leap_gb300.autograd import calibrate_lm  # noqa: E402

DEVICE = "cuda:0"
C_LIGHT = 299792458.0
PHASE_CENTRE = synth.PHASE_CENTRE
FORMS = {"fp64": lg.LEAP_PRECISION_FP64, "mixed": lg.LEAP_PRECISION_MIXED}
DTYPES = {"c64": torch.complex64, "c128": torch.complex128}


def _case(kind, stations, timesteps, channels, directions, form, vis="c64", pols=4, box=0.1, **more):
    return dict(kind=kind, stations=stations, timesteps=timesteps, channels=channels, directions=directions, form=form,
                vis=vis, pols=pols, box=box, **more)


def listed():
    return [
        # The smallest call: one direction on the 36-antenna array, complex<double>, the reference's own types.
        dict(_case("resident", 36, 1, 48, 1, "fp64", vis="c128"), name="askap36_fp64"),
        # A small mixed call, where launches and uploads of tables are what is waited for.
        dict(_case("resident", 24, 2, 32, 6, "mixed"), name="small24_mixed"),
        # One solution interval of one timestep in the default (FP64) form, straight from the MeasurementSet's DATA.
        dict(_case("upload", 128, 1, 384, 64, "fp64", order="ms", memory="host"), name="slice1_host_fp64"),
        # The 128-antenna workload in the all-FP64 form.
        dict(_case("resident", 128, 14, 384, 64, "fp64"), name="mwa128_fp64"),
        # The same in the mixed form: 64 directions, enough for the gridded kernel.
        dict(_case("resident", 128, 14, 384, 64, "mixed"), name="mwa128_mixed"),
        # Nine directions far from the phase centre, as the reference's end-to-end run has.
        dict(_case("resident", 128, 14, 384, 9, "mixed", box=0.9), name="mwa128_9dir_mixed"),
        # Two polarisations held as complex<double> (the reference's Integration type), mixed form.
        dict(_case("resident", 128, 4, 96, 16, "mixed", vis="c128", pols=2), name="c128_2pol_mixed"),
        # A whole observation as one solution interval, from pageable host memory in MeasurementSet order.
        dict(_case("upload", 128, 14, 384, 64, "mixed", order="ms", memory="host"), name="mwa128_host_mixed"),
        # A correlator or simulator on the same GPU hands its integration over.
        dict(_case("upload", 128, 14, 384, 64, "mixed", order="integration", memory="device"), name="mwa128_device_mixed"),
        # The batched workload: 32 uneven chunks, 256 directions, 52 GB.
        dict(_case("batched", 128, 0, 0, 256, "mixed", chunks=32, max_timesteps=64, layout=4), name="batched_uneven"),
        # 512 stations of a low-frequency array, 128 directions.
        dict(_case("resident", 512, 16, 384, 128, "mixed"), name="ska_low_mixed"),
        # Cal phases and their gradients, as an optimiser over directions and visibilities calls them.
        dict(_case("grad", 128, 8, 96, 16, "fp64"), name="grad_fp64"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["resident", "resident", "resident", "upload", "upload", "batched", "grad"])
    stations = _log_int(rng, 16, 160)
    channels = _log_int(rng, 16, 400)
    if kind == "batched":
        return _case(kind, stations, 0, 0, _log_int(rng, 8, 256), "mixed", chunks=rng.randint(2, 16),
                     max_timesteps=_log_int(rng, 2, 48), layout=rng.randint(5, 1000))
    if kind == "grad":
        return _case(kind, stations, rng.randint(1, 8), min(channels, 128), _log_int(rng, 1, 24), "fp64",
                     vis=rng.choice(["c64", "c64", "c128"]), pols=rng.choice([4, 4, 2, 1]))
    form = rng.choice(["fp64", "mixed", "mixed"])
    timesteps = rng.randint(1, 14)
    directions = _log_int(rng, 1, 128 if form == "mixed" else 64)
    vis, pols = rng.choice([("c64", 4), ("c64", 4), ("c64", 4), ("c128", 4), ("c64", 2), ("c128", 2), ("c64", 1)])
    more = {}
    if kind == "upload":
        more = dict(order=rng.choice(["ms", "integration"]), memory=rng.choice(["host", "device"]))
    return _case(kind, stations, timesteps, channels, directions, form, vis=vis, pols=pols, box=rng.choice([0.1, 0.1, 0.9]),
                 **more)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _shape(stations, timesteps, channels, pols, offset):
    """The observation without visibilities: the array, its baselines, UVWs and spectral window."""
    if stations > 256:
        spec, f0, df, sigma = synth.ArraySpec(stations, 40000.0, "loguniform"), 100e6, 5.4e3, 1.0
    elif stations == 36:
        spec, f0, df, sigma = synth.ArraySpec(stations, 3000.0), 700e6, 1e6, 0.1
    else:
        spec, f0, df, sigma = synth.ArraySpec(stations, 1500.0), 150e6, 40e3, 0.5
    return synth.make_observation(spec, timesteps, channels, f0, df, sigma, with_vis=False, timestep_offset=offset, pols=pols)


@functools.lru_cache(maxsize=16)
def _metadata(stations):
    """MetaData of the array (the same for every observation of it; built once by a program)."""
    return lg.build_metadata(_shape(stations, 1, 1, 4, 0))


def _set_metadata(ctx, obs):
    """Phase matrices on the host for small arrays (the class's default), on the device for large ones."""
    if obs.num_stations > 256:
        ctx.build_metadata(obs, fetch=False)
        return
    md = _metadata(obs.num_stations)
    ctx.set_metadata(lg.MetaData(obs.nbaselines, md.reference_antenna, obs.channels, obs.pols, obs.num_stations, obs.rows,
                                 obs.freq_start_hz, obs.freq_inc_hz, obs.phase_centre[0], obs.phase_centre[1],
                                 md.A, md.I, md.Ad, md.A1, md.I1, md.Ad1))


def _visibilities(obs, vis, seed, nans=0):
    """The Integration-order cube (channels, rows, pols) on the GPU: a point source seen through random antenna
    gains, with Gaussian noise; `nans` samples lost by the correlator are NaN."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    gains = torch.exp(1j * 2 * math.pi * torch.rand(obs.num_stations, generator=g, device=DEVICE, dtype=torch.float64))
    a1, a2 = (torch.from_numpy(a).to(DEVICE).long() for a in (obs.antenna1, obs.antenna2))
    gg = (gains[a1] * gains[a2].conj()).repeat(obs.timesteps)
    uvw = torch.from_numpy(obs.uvw).to(DEVICE)
    delay = (uvw @ torch.tensor([0.01, -0.005, math.sqrt(1 - 0.01 ** 2 - 0.005 ** 2) - 1], device=DEVICE, dtype=torch.float64))
    cube = torch.empty((obs.channels, obs.rows, obs.pols), dtype=DTYPES[vis], device=DEVICE)
    for c in range(obs.channels):
        model = gg * torch.exp(2j * math.pi * delay * ((obs.freq_start_hz + c * obs.freq_inc_hz) / C_LIGHT))
        noise = torch.randn((obs.rows, obs.pols), generator=g, device=DEVICE, dtype=cube.dtype)
        cube[c] = model.to(cube.dtype)[:, None] + obs.noise_sigma * noise
    if nans:
        at = torch.randint(0, cube.numel(), (nans,), generator=g, device=DEVICE)
        cube.view(-1)[at] = complex(math.nan, 0.0)
    return cube


def _directions(count, box, seed):
    """(l, m) of the directions, and their (ra, dec)."""
    lm = np.random.default_rng(seed).uniform(-box / 2, box / 2, size=(count, 2))
    if box < 0.5:
        lm[0] = (0.01, -0.005)  # the source itself
    return lm, synth.lm_to_radec(lm[:, 0], lm[:, 1])


def _matrices(radec):
    return np.stack([lg.dd_matrix(PHASE_CENTRE[0], PHASE_CENTRE[1], r, d) for r, d in radec])


def _chunks(case):
    """Observations of a batched case and its work items (slot, first direction, count): directions are dealt
    round-robin to the chunks, as many to each as there are."""
    n, per = case["chunks"], [case["directions"] // case["chunks"] + (i < case["directions"] % case["chunks"])
                              for i in range(case["chunks"])]
    shapes = synth.uneven_chunks(n, seed=case["layout"], t_range=(1, case["max_timesteps"]))
    obs = [_shape(case["stations"], s.timesteps, s.channels, case["pols"], s.timestep_offset) for s in shapes]
    first = np.concatenate([[0], np.cumsum(per)])
    return obs, [(i, int(first[i]), per[i]) for i in range(n) if per[i]]


def _nans(case, obs):
    return obs.rows * obs.channels // 2000 if case["kind"] == "upload" else 0


def prepare(case, seed):
    st = {"case": case, "ctx": lg.Context(0), "form": FORMS[case["form"]]}
    ctx = st["ctx"]
    lm, radec = _directions(case["directions"], case["box"], seed)
    st["dds"] = _matrices(radec)
    if case["kind"] == "batched":
        chunks, st["items"] = _chunks(case)
        _set_metadata(ctx, chunks[0])
        for slot, obs in enumerate(chunks):
            ctx.set_integration(slot, _visibilities(obs, case["vis"], seed * 1000 + slot), torch.from_numpy(obs.uvw).to(DEVICE))
        torch.cuda.empty_cache()
        return st
    obs = _shape(case["stations"], case["timesteps"], case["channels"], case["pols"], 0)
    _set_metadata(ctx, obs)
    vis = _visibilities(obs, case["vis"], seed, _nans(case, obs))
    uvw = torch.from_numpy(obs.uvw).to(DEVICE)
    if case["kind"] == "grad":
        st["lm"] = torch.from_numpy(lm).to(DEVICE).requires_grad_()
        st["vis"], st["uvw"] = vis.requires_grad_(), uvw
        st["weights"] = _weights(case, seed)
    elif case["kind"] == "upload":
        if case["order"] == "ms":
            vis = vis.transpose(0, 1).contiguous()
        st["vis"], st["uvw"] = (vis, uvw) if case["memory"] == "device" else (vis.cpu().numpy(), obs.uvw)
    else:
        ctx.set_integration(0, vis, uvw)
        if case["stations"] > 256:  # a program on device tensors
            st["dds"] = torch.from_numpy(st["dds"].reshape(-1)).to(DEVICE)
            st["cal"] = torch.zeros((case["directions"], case["stations"]), dtype=torch.float64, device=DEVICE)
    del vis
    torch.cuda.empty_cache()
    return st


def _weights(case, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn((case["directions"], case["stations"]), generator=g, dtype=torch.float64).to(DEVICE)


def run(st):
    case, ctx, form = st["case"], st["ctx"], st["form"]
    if case["kind"] == "grad":
        cal = calibrate_lm(ctx, 0, st["lm"], st["vis"], st["uvw"], form)
        g_lm, g_vis = torch.autograd.grad(cal, (st["lm"], st["vis"]), st["weights"])
        return {"cal": cal.detach(), "grad_lm": g_lm, "grad_vis": g_vis}
    if case["kind"] == "batched":
        cal = ctx.calibrate_batched(st["items"], st["dds"], form)
    elif "cal" in st:
        ctx.calibrate_async(0, st["dds"].data_ptr(), case["directions"], form, st["cal"].data_ptr(),
                            torch.cuda.current_stream().cuda_stream)
        return {"cal": st["cal"].to(torch.float32) if case["form"] == "mixed" else st["cal"]}
    else:
        if case["kind"] == "upload":
            (ctx.set_integration_ms if case["order"] == "ms" else ctx.set_integration)(0, st["vis"], st["uvw"])
        cal = ctx.calibrate(0, st["dds"], form)
    return {"cal": cal.astype(np.float32) if case["form"] == "mixed" else cal}


def work(case):
    """Each visibility and UVW read once, each result written once; a complex multiply-add (8 operations) per
    sample and direction."""
    sample = 8 if case["vis"] == "c64" else 16
    parts = [(o.rows * o.channels, o.rows, n) for o, (_, _, n) in zip(*_chunk_pairs(case))]
    samples = sum(g for g, _, _ in parts) * case["pols"]
    nbytes = samples * sample + sum(r for _, r, _ in parts) * 24 + case["directions"] * case["stations"] * 8
    flops = sum(g * n for g, _, n in parts) * case["pols"] * 8
    if case["kind"] == "grad":  # the gradient of the visibilities, and the backward sums over pol 0
        nbytes += samples * sample
        flops += 2 * flops // case["pols"]
    return {"bytes": nbytes, "flops": flops}


def _chunk_pairs(case):
    if case["kind"] == "batched":
        obs, items = _chunks(case)
        return [obs[i] for i, _, _ in items], items
    return [_shape(case["stations"], case["timesteps"], case["channels"], case["pols"], 0)], [(0, 0, case["directions"])]


# ---------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ---------------------------------------------------------------------------

def _solver(obs):
    """Baseline lists of the two phase matrices, and x -> pinv(A) x for a given list.  Every row of A is +1 / -1
    for a baseline's antennas; the last row fixes the phase of one antenna.  A has full column rank, so its
    pseudo-inverse is inv(A'A) A' (one step of refinement takes the inverse's rounding out)."""
    S, ref = obs.num_stations, obs.num_stations - 1
    a1, a2 = (torch.from_numpy(a).to(DEVICE).long() for a in (obs.antenna1, obs.antenna2))
    cross = (a1 != a2) & (torch.from_numpy(obs.flags).to(DEVICE) == 0)

    def pinv(rows, fixed):
        p, q = a1[rows], a2[rows]
        G = torch.zeros((S, S), dtype=torch.float64, device=DEVICE)
        one = torch.ones(len(rows), dtype=torch.float64, device=DEVICE)
        for i, j, s in ((p, p, 1), (q, q, 1), (p, q, -1), (q, p, -1)):
            G.index_put_((i, j), s * one, accumulate=True)
        G[fixed, fixed] += 1
        Gi = torch.linalg.inv(G)
        Gi = Gi + Gi @ (torch.eye(S, dtype=torch.float64, device=DEVICE) - G @ Gi)

        def apply(y):  # y: (D, rows), the fixed row's entry is 0
            b = torch.zeros((y.shape[0], S), dtype=torch.float64, device=DEVICE)
            b.index_add_(1, p, y)
            b.index_add_(1, q, y, alpha=-1)
            x = b @ Gi.T
            return x + (b - x @ G.T) @ Gi.T
        return apply

    I = torch.nonzero(cross)[:, 0]
    I1 = torch.nonzero(cross & ((a1 == ref) | (a2 == ref)))[:, 0]
    return a1[I], a2[I], len(I), I1, pinv(I, 0), pinv(I1, ref)


def _average(obs, v0, l, m, n):
    """Pol 0 of one direction's averages over channels and timesteps."""
    uvw = torch.from_numpy(obs.uvw).to(DEVICE)
    shift = -2 * math.pi * ((uvw[:, 0] * l + uvw[:, 1] * m + uvw[:, 2] * n) - uvw[:, 2])
    lam = C_LIGHT / (obs.freq_start_hz + torch.arange(obs.channels, dtype=torch.float64, device=DEVICE) * obs.freq_inc_hz)
    total = torch.zeros(obs.nbaselines, dtype=torch.complex128, device=DEVICE)
    for t in range(obs.timesteps):
        r = slice(t * obs.nbaselines, (t + 1) * obs.nbaselines)
        phase = shift[None, r] / lam[:, None]
        total = total + (v0[:, r] * torch.complex(torch.cos(phase), torch.sin(phase))).sum(0)
    return total


def _solve(avg, solver):
    a1, a2, nI, I1, pinv, pinv1 = solver
    cal1 = pinv1(torch.angle(avg[:, I1]))
    turns = cal1[:, a1] - cal1[:, a2]
    turned = torch.polar(torch.ones_like(turns), -2 * math.pi * turns) * avg[:, :nI]  # row n of avg, not I[n]
    return pinv(torch.angle(turned)) + cal1


def _pol0(obs, cube):
    v0 = torch.empty(cube.shape[:2], dtype=torch.complex128 if cube.numel() < 1 << 28 else cube.dtype, device=DEVICE)
    for c in range(obs.channels):
        bad = torch.isnan(torch.view_as_real(cube[c])).any(-1).any(-1)
        v0[c] = torch.where(bad, torch.zeros((), dtype=cube.dtype, device=DEVICE), cube[c, :, 0])
    return v0


def exact(case, seed):
    lm, radec = _directions(case["directions"], case["box"], seed)
    lmn = torch.from_numpy(_matrices(radec)[:, 2]).to(DEVICE)  # the third rows of the matrices that run() is given
    if case["kind"] == "batched":
        chunks, items = _chunks(case)
        solver = _solver(chunks[0])
        cal = torch.zeros((case["directions"], case["stations"]), dtype=torch.float64, device=DEVICE)
        for slot, d0, nd in items:
            v0 = _pol0(chunks[slot], _visibilities(chunks[slot], case["vis"], seed * 1000 + slot))
            avg = torch.stack([_average(chunks[slot], v0, *lmn[d]) for d in range(d0, d0 + nd)])
            cal[d0:d0 + nd] = _solve(avg, solver)
        return {"cal": cal}
    obs = _shape(case["stations"], case["timesteps"], case["channels"], case["pols"], 0)
    cube = _visibilities(obs, case["vis"], seed, _nans(case, obs))
    v0 = _pol0(obs, cube)
    if case["kind"] != "grad":
        del cube
        return {"cal": _solve(torch.stack([_average(obs, v0, *x) for x in lmn]), _solver(obs))}
    weights, solver, cals = _weights(case, seed), _solver(obs), []
    lm = torch.from_numpy(lm).to(DEVICE)
    g_lm, g_v0 = torch.zeros_like(lm), torch.zeros_like(v0)
    for d in range(case["directions"]):
        x, v = lm[d].clone().requires_grad_(), v0.detach().requires_grad_()
        cal = _solve(_average(obs, v, x[0], x[1], torch.sqrt(1 - x[0] * x[0] - x[1] * x[1]))[None], solver)
        cals.append(cal.detach())
        gx, gv = torch.autograd.grad(cal, (x, v), weights[d:d + 1])
        g_lm[d] = gx
        g_v0 += gv
    g_vis = torch.zeros(cube.shape, dtype=torch.complex128, device=DEVICE)
    g_vis[:, :, 0] = g_v0
    return {"cal": torch.cat(cals), "grad_lm": g_lm, "grad_vis": g_vis}
