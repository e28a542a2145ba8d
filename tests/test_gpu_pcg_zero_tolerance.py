"""The one-launch multigrid PCG past convergence: with tolerance 0 its recursive residual falls until its squares are
subnormal, and the direction stays.

Bar: the steps past a relative residual of 1e-12 change the direction by less than the suite's bar for two solves at that
tolerance, 1e-8 of the largest entry."""
import ctypes

import pytest
import torch

from fastipc_gb300 import _native as N
from fastipc_gb300 import scenes
from fastipc_gb300.newton import NewtonIPC
from test_gpu_pcg_run import SCENES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('fp32', [True, False])
@pytest.mark.parametrize('name,maxit', [('two_cubes_1024', 600), ('two_cubes_1024', 2000), ('bar_thin', 2000), ('pile_small', 4000)])
def test_direction_stays(name, maxit, fp32):
    sim = NewtonIPC(scenes.predeform(SCENES[name](), 5e-5, 3), pcg_rtol=1e-12)
    sim.set_multigrid_fp32(fp32)
    sim.compute_xn_and_xTilde()
    sim.move_nodes(0.0)
    sim.find_constraints()
    sim.compute_hessian_and_gradient()
    sim.solve_system(0.0)
    want = sim.data_sol.clone()
    it = ctypes.c_int()
    st = N.lib().fipc_solve_system(sim.ctx, N.dptr(sim.fixed), ctypes.c_double(0.0), maxit, 0, N.dptr(sim.data_sol), ctypes.byref(it), N.stream())
    assert st in (0, 2)   # the residual became zero, or the budget ran out
    assert torch.isfinite(sim.data_sol).all()
    assert (sim.data_sol - want).abs().max() <= 1e-8 * want.abs().max()
    sim.close()
