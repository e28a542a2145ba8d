"""Constraint rows in closed form and the sums of their blocks, where they can go wrong: gaps from a tenth
to a millionth of the geometry's size (the eigenproblem is graded by the ratio), row counts around the
block size, rows outside the barrier, and runs of more blocks than one group sums (the vertices of a
ground face).

Tolerances.  A row's distance is a difference of coordinates of order one that cancels to the gap s: its
relative error is up to about 10 eps / s on either side, and the barrier's second derivative amplifies it
by about 8 at these distances; slivers and oblique edges (cosines to 0.95) by 10 more: 1e-12 / s bounds both
sides' sum.  Sums of blocks: the bar of the assembled system, 1e-9 of its largest entry."""
import numpy as np
import pytest

from fastipc_gb300.newton import NewtonIPC
from oracle import oracle as O
from tests.test_gpu_broadphase import _touching
from tests.test_gpu_kernels import barrier_gpu

pytestmark = pytest.mark.gpu


def _unit(a):
    return a / np.linalg.norm(a, axis=-1, keepdims=True)


def _rows(t, N, gap, rng):
    """Rows of unit size a distance of about `gap` apart, at every obliqueness and aspect to 1:10."""
    o = rng.uniform(-0.5, 0.5, (N, 3))
    e1 = _unit(rng.normal(size=(N, 3)))
    b = _unit(np.cross(e1, rng.normal(size=(N, 3))))
    n = np.cross(e1, b)
    e2 = rng.uniform(0.1, 1, (N, 1)) * b + rng.uniform(-0.3, 0.3, (N, 1)) * e1
    s = gap * rng.uniform(0.7, 1.3, (N, 1))
    u, v = rng.uniform(0.05, 0.95, (2, N, 1))
    X = np.zeros((N, 4, 3))
    if t == 0:
        X[:, 0], X[:, 1] = o, o + s * n
    elif t == 1:
        X[:, 0], X[:, 1], X[:, 2] = o + u * e1 + s * n, o, o + e1
    elif t == 2:
        v = v * (1 - u)
        X[:, 0], X[:, 1], X[:, 2], X[:, 3] = o + u * e1 + v * e2 + s * n, o, o + e1, o + e2
    else:
        p = o + u * e1 + s * n
        X[:, 0], X[:, 1], X[:, 2], X[:, 3] = o, o + e1, p - v * e2, p + (1 - v) * e2
    return X


def _rel(a, b):
    a, b = a.reshape(len(a), -1), b.reshape(len(b), -1)
    return (np.abs(a - b).max(axis=1) / np.abs(b).max(axis=1)).max()


@pytest.mark.parametrize('gap', [1e-1, 1e-2, 1e-4, 1e-6])
@pytest.mark.parametrize('t,N', [(0, 64), (1, 65), (2, 63), (3, 500), (2, 1)])
def test_graded_rows(t, N, gap):
    X = _rows(t, N, gap, np.random.default_rng(100 * t + N))
    dh2 = (2 * gap) ** 2
    E, g, H = barrier_gpu(t, X, X, dh2, 1e4)
    rows = (np.arange(N)[:, None] * 4 + np.arange(O.TYPE_NV[t])[None, :]).astype(np.int32)
    Eo, go, Ho = O.barrier_rows(t, rows, X.reshape(-1, 3), X.reshape(-1, 3), dh2, 1e4)
    tol = 1e-12 / gap
    np.testing.assert_allclose(E, Eo, rtol=tol)
    assert _rel(g, go) < tol
    assert _rel(H, Ho) < tol


@pytest.mark.parametrize('t', range(4))
def test_negative_stiffness(t):
    """The closed forms' signs are a positive kappa's; others take the general projection."""
    N = 70
    X = _rows(t, N, 0.1, np.random.default_rng(t))
    E, g, H = barrier_gpu(t, X, X, 0.04, -1e4)
    rows = (np.arange(N)[:, None] * 4 + np.arange(O.TYPE_NV[t])[None, :]).astype(np.int32)
    Eo, go, Ho = O.barrier_rows(t, rows, X.reshape(-1, 3), X.reshape(-1, 3), 0.04, -1e4)
    np.testing.assert_allclose(E, Eo, rtol=1e-11)
    assert _rel(g, go) < 1e-11
    assert _rel(H, Ho) < 1e-11


@pytest.mark.parametrize('t', range(4))
def test_rows_outside_the_barrier_are_zero(t):
    E, g, H = barrier_gpu(t, _rows(t, 5, 0.1, np.random.default_rng(t)), np.zeros((5, 4, 3)), 1e-4, 1e4)
    assert not E.any() and not g.any() and not H.any()


@pytest.mark.parametrize('n', [3, 17])
def test_sums_of_long_runs(n):
    """n = 3: no run above 128 blocks; 17: those of the ground's vertices."""
    sc = _touching(n, 0.6, 0.2)
    sim, o = NewtonIPC(sc), O.OracleSim(sc, solver='bsr')
    x = sc.x + np.random.default_rng(n).uniform(-1e-4, 1e-4, sc.x.shape) * ~sc.dirichlet(0.0)[0][:, None]
    sim.set_state(x, np.zeros_like(x))
    o.x, o.v = x.copy(), np.zeros_like(x)
    for q in (sim, o):
        q.compute_xn_and_xTilde()
        q.find_constraints()
        q.compute_hessian_and_gradient()
    runs = {}
    for r in o.rows:
        for row in r:
            for v in row:
                runs[v] = runs.get(v, 0) + 1
    assert (max(runs.values()) > 128) == (n == 17)
    _, act, rhs = sim.export_system()
    assert act.data.shape == (len(o.c_ci), 3, 3)
    np.testing.assert_array_equal(act.indptr, o.c_rp)
    np.testing.assert_array_equal(act.indices, o.c_ci)
    assert np.abs(act.data.reshape(-1, 9) - o.c_va).max() <= 1e-9 * np.abs(o.c_va).max()
    assert np.abs(rhs - o.rhs.ravel()).max() <= 1e-9 * np.abs(o.rhs).max()
    E, Eo = sim.compute_energy(), o.compute_energy()
    assert abs(E - Eo) <= 1e-10 * abs(Eo)
