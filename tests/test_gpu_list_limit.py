"""Queries whose candidate lists are full: pairs past the end of a pair list or a filter list are tested by the lane that found
them.  The lists' counters show that they overflowed.

Bars: constraint lists and intersection flag equal to those without a limit and to the oracle's; the step 1e-12 relative to
either."""
import ctypes

import numpy as np
import pytest
import torch

from fastipc_gb300 import _native as N
from fastipc_gb300 import scenes
from fastipc_gb300.newton import NewtonIPC
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def stats(s):
    out = (ctypes.c_longlong * 10)()
    assert N.lib().fipc_broadphase_stats(s.ctx, out) == 0
    return list(out)


@pytest.fixture(scope='module')
def pile():
    """Two cubes 0.8 contact distances apart and a ground box of a few large triangles 0.8 below them."""
    rng = np.random.default_rng(3)
    dhat = 1e-3
    base, ct = scenes.hex_grid(6, 6, 6, (0.1, 0.1, 0.1))
    ground, gt = scenes.hex_grid(1, 1, 1, (1.0, 0.1, 1.0))
    x = np.concatenate([base + np.array([0.0, 0.8 * dhat, 0.0]), base + np.array([0.013, 0.1 + 1.6 * dhat, 0.017]),
                        ground + np.array([-0.4, -0.1, -0.4])])
    tets = np.concatenate([ct, ct + len(base), gt + 2 * len(base)]).astype(np.int32)
    sc = scenes.Scene('pile', x, tets, np.zeros_like(x), *scenes.find_boundary(tets), None, dhat=dhat, dt=0.01)
    sc.dirichlet = lambda t: (np.arange(len(x)) >= 2 * len(base), x)
    pos = x + rng.uniform(-0.05, 0.05, x.shape) * dhat
    p = rng.uniform(-0.2, 0.2, x.shape) * dhat
    p[:len(base), 1] -= 0.3 * dhat
    p[len(base):2 * len(base), 1] -= 3 * dhat
    p[2 * len(base):] = 0.0
    s, o = NewtonIPC(sc), O.OracleSim(sc, solver='bsr')
    hit = pos + 1.5 * p

    def run():
        s.x.copy_(torch.from_numpy(pos))
        s.data_sol.copy_(torch.from_numpy(p))
        s.find_constraints()
        out = [[r.copy() for r in s.constraints()], stats(s)[:2]]
        out += [s.compute_intersection_free_step_size(), stats(s)[:4]]
        out += [s.check_collision(), stats(s)[:1]]
        s.x.copy_(torch.from_numpy(hit))
        return out + [s.check_collision()]

    free = run()
    o.x = pos.copy()
    o.find_constraints()
    for got, want in zip(free[0], o.rows):
        np.testing.assert_array_equal(got, want)
    alpha = o.compute_intersection_free_step_size(p)
    assert alpha < 1.0 and abs(free[2] - alpha) <= 1e-12 * alpha
    assert free[4] == o.check_collision() == False  # noqa: E712
    o.x = hit.copy()
    assert free[6] == o.check_collision() == True  # noqa: E712
    yield s, run, free
    s.close()


@pytest.mark.parametrize('limit', [0, 1, 33, 100])
def test_full_lists(pile, limit):
    s, run, free = pile
    assert min(free[1]) > 100 and min(free[3]) > 100 and free[5][0] > 100   # every list is longer than every limit
    assert N.lib().fipc_ctx_set_list_limit(s.ctx, limit) == 0
    try:
        got = run()
    finally:
        assert N.lib().fipc_ctx_set_list_limit(s.ctx, -1) == 0
    for a, b in zip(got[0], free[0]):
        np.testing.assert_array_equal(a, b)
    assert abs(got[2] - free[2]) <= 1e-12 * free[2] and got[4] == free[4] and got[6] == free[6]
    # a pair list's counter stops at its end; that of a filter list counts all pairs that pass the bound
    assert min(got[1]) >= limit and min(got[3][:2]) >= limit and got[5][0] >= limit
    assert got[3][2:] == free[3][2:]


def test_limit_is_checked(pile):
    assert N.lib().fipc_ctx_set_list_limit(pile[0].ctx, -2) == 5
