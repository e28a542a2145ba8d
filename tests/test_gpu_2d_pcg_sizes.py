"""The 2D PCG around the rules that choose its launch: a few rows, around 32 rows per SM (16 rows per CTA more),
the last size of the cooperative launch and one beyond it, and rows of more blocks than
the lanes keep in shared memory.

Bar: the recursion stops at |r| <= 1e-12 |b|; the true residual differs by the rounding of the iterates, a few
eps (|A| |x| + |b|) per direction of new size: 1e-11 of that (infinity norms)."""
import numpy as np
import pytest
import scipy.sparse.linalg
import torch

from fastipc_gb300 import scenes
from fastipc_gb300.newton2d import NewtonIPC2D

pytestmark = pytest.mark.gpu


def _solve(sc, seed, size):
    sim = NewtonIPC2D(sc, pcg_rtol=1e-12)
    x = sc.x + np.random.default_rng(seed).uniform(-size, size, sc.x.shape) * ~sc.dirichlet(0.0)[0][:, None]
    sim.set_state(x, np.zeros_like(x))
    sim.compute_xn_and_xTilde()
    sim.move_nodes(0.0)
    sim.find_constraints()
    sim.compute_hessian_and_gradient()
    A, b = sim.export_system()
    A = A.tocsr()
    sim.solve_system(0.0)
    y = sim.data_sol.cpu().numpy().ravel()
    fixed = np.repeat(sim.fixed.cpu().numpy().ravel().astype(bool), 2)
    assert not y[fixed].any()
    free = np.flatnonzero(~fixed)
    A, b, y = A[free][:, free], b[free], y[free]
    r = np.abs(A @ y - b).max()
    assert r <= 1e-11 * (scipy.sparse.linalg.norm(A, np.inf) * np.abs(y).max() + np.abs(b).max()), r
    assert 0 < sim.pcg_iters[-1] < 20000
    first = sim.data_sol.clone()
    sim.solve_system(0.0)
    assert torch.equal(first, sim.data_sol)      # every sum in a fixed order


@pytest.mark.parametrize('k,n', [(1, 1), (1, 3), (16, 16), (17, 16)])
def test_sizes(k, n):
    _solve(scenes.square_stack_2d(k, n), k, 2e-4)


@pytest.mark.parametrize('k', [40, 41])
def test_last_size_of_one_launch(k):
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    sc = scenes.square_stack_2d(k, 30)
    assert (len(sc.x) <= 256 * sm) == (k == 40) or sm != 152
    _solve(sc, k, 1e-4)


@pytest.mark.parametrize('rim', [15, 16, 33, 100])
def test_rows_of_many_blocks(rim):
    """A fan: its centre's row has rim + 1 blocks."""
    t = 2 * np.pi * np.arange(rim) / rim
    x = np.concatenate([[[0.0, 0.5]], np.stack([0.1 * np.cos(t), 0.5 + 0.1 * np.sin(t)], 1)])
    tris = np.stack([np.zeros(rim, int), 1 + np.arange(rim), 1 + (np.arange(rim) + 1) % rim], 1).astype(np.int32)
    bp, be = scenes.find_boundary_2d(tris)
    mask = np.zeros(len(x), bool)
    _solve(scenes.Scene2D('fan', x, tris, np.zeros_like(x), bp, be, lambda t: (mask, x), steps=1, meta={}), rim, 1e-4)
