"""The gridded kernel's way out when a wait gives up, modelled on the CPU.

A role that a whole warp walks (MMA issuer, fold and epilogue warps of csrc/kernels_grid.cuh) has shuffles, warp barriers
and warp-wide tcgen05 instructions after its waits, which every lane of the warp must reach.  Each lane polls a wait on
its own, and the abort flag that another role raises may be seen by some lanes before the phase completes, by others
after.  The model polls 32 lanes in random order while an abort and a completion land at random times, joins the lanes'
outcomes as the wait function that the kernel's role calls does, and checks that all lanes take the same way."""
import os
import random
import re

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "icrar-leap-accelerate_gb300",
                      "csrc", "kernels_grid.cuh")
LANES = 32


def _source():
    return open(HEADER).read()


def _role(name):
    """The source of a role: from its heading to the next one's, or to the block's closing barrier."""
    text = _source()
    begin = text.index("// ---------------- %s" % name)
    ends = [i for i in (text.find("// ----------------", begin + 20), text.find("__syncthreads();", begin)) if i >= 0]
    return text[begin:min(ends)]


def _votes(function):
    """Whether a wait function joins its lanes' outcomes."""
    m = re.search(r"bool %s\(.*?\n}" % function, _source(), re.S)
    assert m, function
    return "__all_sync(0xffffffffu" in m.group(0)


def lane_outcomes(rng):
    """Each lane's own outcome of one wait: lanes poll in any order, look at the abort flag at every 4th poll of theirs,
    and the phase completes and the abort lands at random times."""
    complete, abort = rng.randint(0, 600), rng.randint(0, 600)
    polls, out, clock = [0] * LANES, [None] * LANES, 0
    while None in out:
        lane = rng.choice([i for i in range(LANES) if out[i] is None])
        clock += 1
        polls[lane] += 1
        if clock >= complete:
            out[lane] = True
        elif polls[lane] % 4 == 0 and clock >= abort:
            out[lane] = False
    return out


def diverges(votes, seed):
    rng = random.Random(seed)
    for _ in range(200):
        out = lane_outcomes(rng)
        if votes:
            out = [all(out)] * LANES
        if len(set(out)) > 1:
            return True
    return False


@pytest.mark.parametrize("role,waits", [("MMA issuer", 4), ("fold warps", 3), ("epilogue", 1)])
def test_lanes_leave_together(role, waits):
    text = _role(role)
    calls = re.findall(r"!(grid_wait\w*)\(", text)
    assert len(calls) == waits, calls
    assert re.search(r"__syncwarp\(\)|_sync\(|sync\.aligned|grid_uniform|grid_fold", text)  # lanes must stay together
    for function in set(calls):
        assert not diverges(_votes(function), 1), function


def test_the_model_tells_a_wait_without_a_vote():
    assert diverges(False, 2)
