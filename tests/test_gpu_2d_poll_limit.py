"""A 2D solve whose one-launch PCG gives up waiting (a limit of 0 reads: the first exchange does) is done by the separate
kernels.

Bar: as in test_gpu_2d_pcg_sizes.py for the two solutions' difference through the system: both meet
|A y - b| <= 1e-11 (|A| |y| + |b|)."""
import numpy as np
import pytest
import scipy.sparse.linalg
import torch

from fastipc_gb300 import _native as N
from fastipc_gb300 import scenes
from fastipc_gb300.newton2d import NewtonIPC2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('k,n', [(1, 3), (16, 16)])
def test_falls_through(k, n):
    sc = scenes.square_stack_2d(k, n)
    sim = NewtonIPC2D(sc, pcg_rtol=1e-12)
    x = sc.x + np.random.default_rng(k).uniform(-2e-4, 2e-4, sc.x.shape) * ~sc.dirichlet(0.0)[0][:, None]
    sim.set_state(x, np.zeros_like(x))
    sim.compute_xn_and_xTilde()
    sim.move_nodes(0.0)
    sim.find_constraints()
    sim.compute_hessian_and_gradient()
    A, b = sim.export_system()
    fixed = np.repeat(sim.fixed.cpu().numpy().ravel().astype(bool), 2)
    free = np.flatnonzero(~fixed)
    A, b = A.tocsr()[free][:, free], b[free]
    launches = []
    for limit in (1 << 20, 0, 1 << 20):
        assert N.lib().fipc2d_ctx_set_poll_limit(sim.ctx, limit) == 0
        sim.data_sol.fill_(7.0)
        n0 = N.launch_count()
        sim.solve_system(0.0)
        launches.append(N.launch_count() - n0)
        y = sim.data_sol.cpu().numpy().ravel()
        assert not y[fixed].any()
        y = y[free]
        assert np.abs(A @ y - b).max() <= 1e-11 * (scipy.sparse.linalg.norm(A, np.inf) * np.abs(y).max() + np.abs(b).max())
        assert sim.pcg_iters[-1] > 0
    assert launches[0] == launches[2] == 1 and launches[1] > 3 * sim.pcg_iters[1]
    assert N.lib().fipc2d_ctx_set_poll_limit(sim.ctx, -1) == 5
    torch.cuda.synchronize()
