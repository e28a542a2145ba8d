"""The hash table, the big-primitive pass and the two row sorts at their edges, against the oracle (which
hashes every primitive): lists exact, CCD step 1e-12 relative, intersection flag equal.

Sizes: a few rows and around 2,048 (the one-CTA sort's limit), repeated calls on a context whose table
and row buffers have to grow, and states whose moving boxes cover many cells (every primitive big)."""
import numpy as np
import pytest
import torch

from fastipc_gb300 import scenes
from fastipc_gb300.newton import NewtonIPC
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _touching(n, gap, turn, ground=True):
    """Two cubes of n hexes a side, `gap` contact distances apart, over a ground box."""
    base, tets = scenes.hex_grid(n, n, n, (0.1, 0.1, 0.1))
    R = scenes.rotation_matrix((0, 1, 0), turn)
    parts = [(base - 0.05 + [0, 0.05 + gap * 1e-3, 0], tets), ((base - 0.05) @ R.T + [0, 0.15 + 2 * gap * 1e-3, 0], tets)]
    mask = np.zeros(2 * len(base), bool)
    if ground:
        g, gt = scenes.hex_grid(1, 1, 1, (0.6, 0.1, 0.6))
        parts.append((g - [0.3, 0.1, 0.3], gt))
        mask = np.concatenate([mask, np.ones(len(g), bool)])
    return scenes._finish('touching', parts, np.zeros((len(mask), 3)), scenes._static_dirichlet(mask), script=scenes._static_script(mask))


def _check(sim, o, x, p):
    sim.set_state(x, np.zeros_like(x))
    o.x = x.copy()
    sim.find_constraints()
    o.find_constraints()
    rows = sim.constraints()
    for t in range(7):
        np.testing.assert_array_equal(rows[t], o.rows[t], err_msg=f'list {t}')
    assert sim.check_collision() == bool(o.check_collision())
    sim.data_sol.copy_(torch.from_numpy(p))
    a, ref = sim.compute_intersection_free_step_size(), o.compute_intersection_free_step_size(p)
    assert abs(a - ref) <= 1e-12 * ref, (a, ref)
    return sum(len(r) for r in rows)


@pytest.mark.parametrize('n,turn,ground', [(1, 0.0, True), (2, 0.3, True), (5, 0.2, False), (9, 0.25, True), (13, 0.1, True), (17, 0.2, True)])
def test_lists_steps_and_flags(n, turn, ground):
    sc = _touching(n, 0.8, turn, ground)
    sim, o = NewtonIPC(sc), O.OracleSim(sc, solver='bsr')
    rng = np.random.default_rng(n)
    fixed = sc.dirichlet(0.0)[0]
    free = ~fixed[:, None]
    x = sc.x + rng.uniform(-1e-4, 1e-4, sc.x.shape) * free
    down = np.zeros_like(x)
    down[:, 1] = -1.0
    n_rows = _check(sim, o, x, (2e-3 * down + rng.uniform(-1e-4, 1e-4, x.shape)) * free)
    assert n_rows > 0 and (n < 17 or n_rows > 2048) and (n > 5 or n_rows < 2048)
    # no contact, then contact again: buffers of another call
    apart = x.copy()
    apart[:, 1] += 0.05 * (np.arange(len(x)) // (n + 1) ** 3) * free[:, 0]
    _check(sim, o, apart, 1e-3 * down * free)
    _check(sim, o, x, rng.uniform(-3e-4, 3e-4, x.shape) * free)
    # long moves: boxes over many cells, most primitives tested outside the grid
    if n <= 5:
        _check(sim, o, x, (0.3 * down + rng.uniform(-0.02, 0.02, x.shape)) * free)
    # an intersecting state
    pushed = x.copy()
    pushed[len(x) - 8 * ground - (n + 1) ** 3:len(x) - 8 * ground, 1] -= 0.021
    sim.set_state(pushed, np.zeros_like(x))
    o.x = pushed.copy()
    assert sim.check_collision() and o.check_collision()
    sim.close()
