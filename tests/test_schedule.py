"""Unit schedule of the persistent kernels (schedule_units in csrc/host_math.cc): every unit once, each block's list
without gaps, one closing round, and the longest block no longer than by giving the units one by one to the least
loaded block."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "icrar-leap-accelerate_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("sched") / "libsched.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "schedule_check.cc"), os.path.join(CSRC, "host_math.cc"), "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)
    lib.schedule_check.restype = lib.greedy_makespan.restype = ctypes.c_longlong
    return lib


# (groups, slabs per group, cost of a full slab, cost of the last slab) of each item
@pytest.mark.parametrize("items", [[(1, 1, 5, 5)], [(7, 1, 26, 26)], [(152, 3, 26, 13)], [(2064, 2, 52, 27), (9, 1, 400, 400)],
                                   [(5, 4, 100, 7), (33, 2, 64, 64), (1, 1, 1, 1)], [(65664, 1, 104, 104)]])
@pytest.mark.parametrize("blocks", [1, 3, 152])
def test_schedule(lib, items, blocks):
    cost, shape, begin = [], [], 0
    for groups, slabs, full, last in items:
        if slabs > 1:
            cost.append(full)
            shape.append((begin, groups * (slabs - 1), slabs - 1, slabs))
        cost.append(last)
        shape.append((begin + slabs - 1, groups, 1, slabs))
        begin += groups * slabs
    cost, shape = np.array(cost, np.int64), np.array(shape, np.int32)
    grid = min(blocks, begin)
    out = np.full(4 * (begin + 2 * grid), -7, np.int32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    size = lib.schedule_check(len(cost), p(cost), p(shape), grid, p(out), ctypes.c_longlong(out.size))
    assert size > 0 and size % grid == 0
    order = out[:size].reshape(-1, grid)
    assert (order[-1] == -1).all() and (order[:-1].max(axis=1) >= 0).all()
    assert sorted(order[order >= 0]) == list(range(begin))
    assert all((np.diff((order[:, b] >= 0).astype(int)) <= 0).all() for b in range(grid))
    unit_cost = np.empty(begin, np.int64)
    for c, (b0, count, per, stride) in zip(cost, shape):
        i = np.arange(count)
        unit_cost[b0 + i // per * stride + i % per] = c
    load = np.where(order >= 0, unit_cost[order], 0).sum(axis=0)
    assert load.max() <= lib.greedy_makespan(len(cost), p(cost), p(shape), grid)
