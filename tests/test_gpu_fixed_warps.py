"""All-FP64 rotate + average: the rule that chooses 1, 2 or 4 warps per block by pols, directions and the call's size,
on both sides of each of its lines, against the oracle (test_gpu_fixed.py's bounds); and calls of many timesteps, whose
slabs are of few or of single timesteps."""
import numpy as np
import pytest

from test_gpu_fixed import _case, _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("pols,stations,timesteps,channels,directions", [
    (4, 6, 1, 20, 2), (4, 6, 1, 20, 3), (4, 6, 2, 20, 12), (4, 33, 7, 17, 9), (4, 33, 6, 17, 9), (4, 33, 5, 17, 17), (4, 33, 7, 3, 4),
    (2, 33, 7, 17, 2), (2, 9, 2, 18, 12), (1, 33, 5, 17, 1), (1, 9, 2, 18, 6)])
def test_warps(ctx, dtype, pols, stations, timesteps, channels, directions):
    _check(ctx, *_case(stations, timesteps, channels, pols, directions, dtype, seed=directions))


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("pols,stations,timesteps,channels,directions", [
    (4, 4, 33, 40, 1), (4, 3, 200, 20, 1), (2, 4, 65, 150, 3), (1, 12, 130, 9, 2), (4, 20, 37, 17, 5)])
def test_many_timesteps(ctx, dtype, pols, stations, timesteps, channels, directions):
    _check(ctx, *_case(stations, timesteps, channels, pols, directions, dtype, seed=timesteps))
