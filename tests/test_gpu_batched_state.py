"""A repeated batched call answers for what the slots, the metadata and the options hold when it is made: each change
between two equal calls that a recorded call could miss, in the pipelined, gridded and FP64 kernels.

Tolerance: that of the form (1e-5 rad mixed, 1e-10 rad FP64) against the oracle on the present data; the averages' is
the same times the size of their terms.  A call after that, with nothing in between, gives the same bits."""
import numpy as np
import pytest
import torch

import oracle
import leap_gb300 as lg
from leap_gb300 import _abi
from leap_gb300.autograd import calibrate_lm
from test_gpu_batched import make_chunks

pytestmark = pytest.mark.gpu

MIXED, FP64 = lg.LEAP_PRECISION_MIXED, lg.LEAP_PRECISION_FP64
FORMS = {"pipelined": (MIXED, [8, 6, 8]), "gridded": (MIXED, [32, 40, 33]), "fp64": (FP64, [3, 8, 1])}
SHAPES = [(3, 48), (1, 96), (5, 20)]


class Batch:
    """Three slots of uneven shape, and the batched call over them."""

    def __init__(self, ctx, form):
        self.ctx = ctx
        self.precision, counts = FORMS[form]
        self.chunks = make_chunks(34, [(t, c, n) for (t, c), n in zip(SHAPES, counts)])
        self.obs = [c[0] for c in self.chunks]
        pc = self.obs[0].phase_centre
        self.dds = np.stack([lg.dd_matrix(*pc, r, d) for _, dirs, _ in self.chunks for r, d in dirs])
        self.items = [(slot, d0, len(dirs)) for slot, (_, dirs, d0) in enumerate(self.chunks)]
        self.upload(ctx)

    def upload(self, ctx):
        ctx.set_metadata(lg.build_metadata(self.obs[0]))
        for slot, obs in enumerate(self.obs):
            ctx.set_integration(slot, obs.vis, obs.uvw)

    def call(self):
        return self.ctx.calibrate_batched(self.items, self.dds, self.precision)

    def check(self):
        cal = self.call()
        tol = 1e-5 if self.precision == MIXED else 1e-10
        mdo = oracle.metadata(self.obs[0])
        for (slot, d0, n), obs in zip(self.items, self.obs):
            exp = oracle.calibrate_interval(obs.vis, obs.uvw, self.dds[d0:d0 + n], mdo)
            assert np.abs(cal[d0:d0 + n] - exp).max() <= tol, slot
            self.ctx._last_slot = slot
            avg = self.ctx.avgdata(d0)
            ref = oracle.rotate_visibilities(obs.vis, obs.uvw, self.dds[d0], obs.nbaselines, obs.freq_start_hz, obs.freq_inc_hz)
            assert np.abs(avg - ref).max() <= tol * np.abs(obs.vis).sum() / obs.nbaselines
        np.testing.assert_array_equal(cal, self.call())  # and once more


@pytest.fixture(params=list(FORMS))
def batch(request):
    with lg.Context(0) as ctx:
        b = Batch(ctx, request.param)
        b.check()
        yield b


def test_other_visibilities(batch):
    obs = batch.obs[1]
    phase = np.random.default_rng(1).uniform(-2, 2, obs.num_stations)
    turn = np.tile(np.exp(1j * (phase[obs.antenna1] - phase[obs.antenna2])), obs.timesteps)
    obs.vis = (obs.vis * turn[None, :, None]).astype(np.complex64)
    batch.ctx.set_integration(1, obs.vis, obs.uvw)
    batch.check()


def test_other_uvws_in_measurementset_order(batch):
    obs = batch.obs[0]
    obs.uvw = obs.uvw * 0.97
    batch.ctx.set_integration_ms(0, np.ascontiguousarray(obs.vis.transpose(1, 0, 2)), obs.uvw)
    batch.check()


def test_flags(batch):
    obs = batch.obs[2]
    flags = (np.random.default_rng(2).uniform(size=(obs.rows, obs.channels, 1)) < 0.4).astype(np.uint8)
    assert batch.ctx.apply_flags(2, flags) == flags.sum()
    obs.vis = np.where(flags[:, :, 0].T[:, :, None] != 0, 0, obs.vis).astype(np.complex64)
    batch.check()


@pytest.mark.parametrize("precision,directions", [(MIXED, 5), (MIXED, 45), (FP64, 4)])
def test_a_single_call_of_another_shape(batch, precision, directions):
    """Fewer channels, timesteps and directions than the slots of the batch, so that no buffer grows."""
    obs = batch.obs[0]
    n = obs.nbaselines
    batch.ctx.set_integration(7, np.ascontiguousarray(obs.vis[:9, :n]), obs.uvw[:n])
    batch.check()
    batch.ctx.calibrate(7, batch.dds[np.arange(directions) % len(batch.dds)], precision)
    batch.check()


def test_another_batch(batch):
    batch.ctx.calibrate_batched([(2, 0, 1), (0, 1, 2)], batch.dds[:3], batch.precision)
    batch.check()
    batch.ctx.set_option(_abi.LEAP_OPTION_GRAPH_REPLAY, 0)
    batch.ctx.calibrate_batched([(2, 0, 1), (0, 1, 2)], batch.dds[:3], batch.precision)
    batch.ctx.set_option(_abi.LEAP_OPTION_GRAPH_REPLAY, 1)
    batch.check()


def test_gradients_of_another_spectral_length(batch):
    obs = batch.obs[0]
    vis = torch.from_numpy(np.ascontiguousarray(obs.vis[:7])).cuda().requires_grad_()
    lm = torch.tensor([[0.01, 0.02], [-0.02, 0.0]], dtype=torch.float64, device="cuda", requires_grad=True)
    calibrate_lm(batch.ctx, 8, lm, vis, torch.from_numpy(obs.uvw).cuda(), FP64).sum().backward()
    batch.check()


def test_another_frequency(batch):
    for obs in batch.obs:
        obs.freq_start_hz, obs.freq_inc_hz = 151.7e6, 37e3
    batch.ctx.set_metadata(lg.build_metadata(batch.obs[0]))
    batch.check()


def test_smaller_integrations(batch):
    """A slot refilled with fewer timesteps, one with fewer channels; then the first again."""
    obs, full = batch.obs, [(o.vis, o.uvw, o.timesteps, o.channels) for o in batch.obs]
    n = obs[0].nbaselines
    obs[0].vis, obs[0].uvw, obs[0].timesteps = np.ascontiguousarray(obs[0].vis[:, :2 * n]), obs[0].uvw[:2 * n], 2
    obs[1].vis, obs[1].channels = np.ascontiguousarray(obs[1].vis[:50]), 50
    for slot in (0, 1):
        batch.ctx.set_integration(slot, obs[slot].vis, obs[slot].uvw)
    batch.check()
    for slot in (0, 1):
        obs[slot].vis, obs[slot].uvw, obs[slot].timesteps, obs[slot].channels = full[slot]
        batch.ctx.set_integration(slot, obs[slot].vis, obs[slot].uvw)
    batch.check()


def test_fewer_baselines_and_stations(batch):
    """Metadata of a smaller array, and its integrations in the same slots."""
    counts = [n for _, _, n in batch.items]
    small = make_chunks(20, [(t, c, n) for (t, c), n in zip(SHAPES, counts)], seed=3)
    batch.obs = [c[0] for c in small]
    batch.upload(batch.ctx)
    batch.check()


def test_released_slot_is_refused(batch):
    batch.ctx.release_integration(1)
    with pytest.raises(lg.LeapError):
        batch.call()
    batch.upload(batch.ctx)
    batch.check()
