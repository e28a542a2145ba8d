"""Triangles and edges of 65 to 256 hash cells leave the grid while few do (their number times the primitives of their
scene) and stay in it otherwise: a body that moves many cells per step, a few vertices that do, and a plate of coarse
edges beside a finer cube.

Bars: the counters say which side of the line a query took; constraint lists exact; CCD step 1e-12 relative; intersection
flag equal to the oracle's, which hashes every primitive."""
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
    return list(out)[:8]


def cell_of(sc):
    e = sc.boundary_edges.reshape(-1, 2)
    return np.median(np.linalg.norm(sc.x[e[:, 0]] - sc.x[e[:, 1]], axis=1))


@pytest.mark.parametrize('n,moving,stay', [(8, 'body', False), (18, 'body', True), (18, 'few', False)])
@pytest.mark.parametrize('u,d', [(20, (0.0, -1.0, 0.0)), (2.5, (-1.0, -1.0, 1.0))])
def test_step_filter(n, moving, stay, u, d):
    sc = scenes.two_cubes(n=n, seed=1)
    s = NewtonIPC(sc)
    o = O.OracleSim(sc, solver='bsr')
    half = len(sc.x) // 2
    mv = np.arange(len(sc.x)) >= half
    if moving == 'few':
        mv &= np.argsort(np.argsort(sc.x[:, 1] + 1e3 * ~mv)) < 12
    # vertices off the lattice: rounding decides the interval test of exactly parallel edges that move together
    rng, cell = np.random.default_rng(n), cell_of(sc)
    x = sc.x + rng.uniform(-0.05, 0.05, sc.x.shape) * cell
    p = np.where(mv[:, None], u * cell * np.array(d), 0.0) + rng.uniform(-0.1, 0.1, sc.x.shape) * cell
    s.x.copy_(torch.from_numpy(x))
    o.x = x.copy()
    s.data_sol.copy_(torch.from_numpy(p))
    a, ref = s.compute_intersection_free_step_size(), o.compute_intersection_free_step_size(p)
    st = stats(s)
    assert ref < 1.0 and abs(a - ref) <= 1e-12 * ref
    if stay:
        assert st[7] > 0 and st[5] < 100 and (st[6] > 0) != (st[4] > 100)
    else:
        assert min(st[4:6]) > 0 and st[6:] == [0, 0]
    s.close()


def plate(fine, coarse):
    """A cube of fine hexes 0.8 contact distances above a plate whose edges are some eight of the cube's."""
    cube, ct = scenes.hex_grid(fine, fine, fine, (0.1, 0.1, 0.1))
    h = 8.0 * 0.1 / fine
    base, bt = scenes.hex_grid(coarse, 1, coarse, (coarse * h, 0.1, coarse * h))
    dhat = 0.4 * 0.1 / fine
    x = np.concatenate([cube + np.array([0.013, 0.8 * dhat, 0.017]), base + np.array([0.0, -0.1, 0.0])])
    tets = np.concatenate([ct, bt + len(cube)]).astype(np.int32)
    points, edges, tris = scenes.find_boundary(tets)
    return scenes.Scene('plate', x, tets, np.zeros_like(x), points, edges, tris, None, dhat=dhat, dt=0.01)


@pytest.mark.parametrize('fine,coarse,stay', [(16, 3, False), (36, 18, True)])
def test_lists_and_check(fine, coarse, stay):
    sc = plate(fine, coarse)
    sc.dirichlet = lambda t: (np.zeros(len(sc.x), bool), sc.x)
    s = NewtonIPC(sc)
    o = O.OracleSim(sc, solver='bsr')
    x = sc.x + np.random.default_rng(fine).uniform(-0.02, 0.02, sc.x.shape) * sc.dhat
    s.x.copy_(torch.from_numpy(x))
    o.x = x.copy()
    s.find_constraints()
    st = stats(s)
    o.find_constraints()
    assert sum(s.counts) > 0
    for got, want in zip(s.constraints(), o.rows):
        np.testing.assert_array_equal(got, want)
    assert st[7] > 0 if stay else (st[5] > 0 and st[7] == 0)
    assert s.check_collision() == o.check_collision() == False  # noqa: E712
    st = stats(s)
    assert st[7] > 0 if stay else (st[5] > 0 and st[7] == 0)
    x[:(fine + 1) ** 3, 1] -= 3 * sc.dhat
    s.x.copy_(torch.from_numpy(x))
    o.x = x.copy()
    assert s.check_collision() == o.check_collision() == True  # noqa: E712
    s.close()
