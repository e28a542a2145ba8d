"""The direct solve at the sizes where its tiles can go wrong: fronts of one vertex to several panels, last
panels and row chunks of 3 to 64, trees of one and of several heights, with and without Dirichlet vertices
and contact.

Bar: Cholesky of an n x n system has a normwise backward error of at most a few n eps; with n < 3,000 the
residual |A x - b| stays below 1e-12 (|A| |x| + |b|) (infinity norms) with a factor of 5 to spare."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg

from fastipc_gb300 import scenes
from fastipc_gb300.newton import NewtonIPC
from tests.test_gpu_broadphase import _touching

pytestmark = pytest.mark.gpu


def _check(sim, x):
    sim.set_state(x, np.zeros_like(x))
    sim.compute_xn_and_xTilde()
    sim.move_nodes(0.0)
    sim.find_constraints()
    sim.compute_hessian_and_gradient()
    A, C, b = sim.export_system()
    A = (A + C).tocsr()
    sim._solve_direct()
    sol = sim.data_sol.cpu().numpy().ravel()
    fixed = np.repeat(sim.fixed.cpu().numpy().ravel().astype(bool), 3)
    assert not sol[fixed].any()
    free = np.flatnonzero(~fixed)
    A, b, y = A[free][:, free], b[free], sol[free]
    r = np.abs(A @ y - b).max()
    assert r <= 1e-12 * (sp.linalg.norm(A, np.inf) * np.abs(y).max() + np.abs(b).max()), r


@pytest.mark.parametrize('size', [(1, 1, 1), (2, 1, 1), (2, 2, 2), (3, 3, 1), (5, 2, 2), (4, 4, 4), (7, 6, 5), (40, 2, 2), (8, 8, 8)])
def test_free_blocks(size):
    x, tets = scenes.hex_grid(*size, (0.02 * size[0], 0.02 * size[1], 0.02 * size[2]))
    mask = np.zeros(len(x), bool)
    sc = scenes._finish('block', [(x, tets)], np.zeros((len(x), 3)), scenes._static_dirichlet(mask), script=scenes._static_script(mask))
    sim = NewtonIPC(sc)
    _check(sim, sc.x + np.random.default_rng(size[0]).uniform(-1e-3, 1e-3, sc.x.shape))


@pytest.mark.parametrize('n', [2, 5])
def test_contact_and_fixed(n):
    sc = _touching(n, 0.7, 0.2)
    sim = NewtonIPC(sc)
    _check(sim, sc.x + np.random.default_rng(n).uniform(-1e-4, 1e-4, sc.x.shape) * ~sc.dirichlet(0.0)[0][:, None])
    assert sum(sim.counts) > 0
