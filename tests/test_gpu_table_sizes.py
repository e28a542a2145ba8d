"""The broad phase's tables after a step filter of a fast step: each query keeps a size of its own, the filter's falls again,
and what the queries return does not depend on what was called before."""
import ctypes

import numpy as np
import pytest
import torch

from fastipc_gb300 import _native as N
from fastipc_gb300 import scenes
from fastipc_gb300.newton import NewtonIPC

pytestmark = pytest.mark.gpu


def slots(s):
    out = (ctypes.c_longlong * 10)()
    assert N.lib().fipc_broadphase_stats(s.ctx, out) == 0
    return out[8], out[9]


def test_sizes_follow_each_query():
    sc = scenes.two_cubes(n=6, seed=2)
    s = NewtonIPC(sc)
    rng = np.random.default_rng(0)
    cell = 0.1 / 6
    s.x.copy_(torch.from_numpy(sc.x + rng.uniform(-0.05, 0.05, sc.x.shape) * cell))
    up = (np.arange(len(sc.x)) >= len(sc.x) // 2)[:, None]
    noise = rng.uniform(-0.1, 0.1, sc.x.shape) * cell
    slow = torch.from_numpy(noise)
    fast = torch.from_numpy(noise + np.where(up, -12.0 * cell, 0.0))

    def step(p):
        s.data_sol.copy_(p)
        return s.compute_intersection_free_step_size(), slots(s)

    def rest():
        s.find_constraints()
        a = [r.copy() for r in s.constraints()], slots(s)
        return a, (s.check_collision(), slots(s))

    first, slow0 = rest(), step(slow)
    fast0 = step(fast)
    assert fast0[1][0] >= 8 * slow0[1][0]
    again = rest()
    for got, want in zip(again[0][0], first[0][0]):
        np.testing.assert_array_equal(got, want)
    assert again[0][1] == first[0][1] and again[1] == first[1]
    for _ in range(24):
        last = step(slow)
        assert last[0] == slow0[0]
    assert last[1][0] <= 4 * slow0[1][0] and last[1][1] <= 4 * slow0[1][1]
    assert step(fast)[0] == fast0[0]
    s.close()
