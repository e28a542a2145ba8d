"""Performance cases: the work that users of this framework have it do, through its public entry points.

A program that uses the framework builds a scene, keeps one simulation object (its context, buffers
and captured graphs) and steps or queries states on it.  So ``prepare`` keeps one object per scene
and makes states (positions, velocities, batches of features) from the seed; ``run`` loads a state
into the object and makes the calls.

Families (``kind``) and what each stands for:

    step        one whole implicit time step (``NewtonIPC.step``) at the default solver tolerance:
                  two cubes about to touch, or a twisted bar in mid-run
    iteration   one Newton iteration by the separate calls of the reference's driver loop (find
                  constraints, system, direction, residual, energy, CCD step, trial point,
                  intersection check, energy at the trial point), solved to 1e-12 as callers that
                  compare with the reference's exact solve do: a pile in contact, or a bar
    constraints the contact lists of a state, fetched to the host
    batch       one Newton iteration of many uneven scenes in one context (``BatchNewtonIPC``)
    direct      the assembled system solved by factorisation instead of PCG
    step2d      one whole 2D time step of a settled column of squares, solved to 1e-12
    admm        two iterations of the ADMM variant of the time step
    train       one optimiser step of the learned warm start on a mini-batch
    infer       the learned warm start's network over a scene's vertices
"""
from functools import lru_cache

import numpy as np
import torch

from fastipc_gb300 import scenes
from fastipc_gb300.admm import AdmmIPC
from fastipc_gb300.batch import BatchNewtonIPC
from fastipc_gb300.learned import WarmStartMLP
from fastipc_gb300.newton import NewtonIPC
from fastipc_gb300.newton2d import NewtonIPC2D

DEV = 'cuda:0'
DT = 0.01
DHAT = 1e-3        # contact distance of the cube scenes
GAP = 0.8          # gap of touching bodies, in units of the contact distance
BAR_STEP = 11      # the bar's cases are in mid-run: 0.11 s after the twist began


def listed():
    return [
        # the smallest 3D scene of the repository's configurations: latencies and launches count
        {'name': 'step_two_cubes', 'kind': 'step', 'scene': 'cubes', 'n': 8},
        # the headline workload, and the largest: 960,000 tets
        {'name': 'step_bar_960k', 'kind': 'step', 'scene': 'bar', 'nx': 400, 'ny': 20, 'nz': 20},
        # an ordinary elastic scene with odd sizes (no contact)
        {'name': 'iteration_bar', 'kind': 'iteration', 'scene': 'bar', 'nx': 101, 'ny': 13, 'nz': 17},
        # 180 cubes settled on one another: contact everywhere, about the size of the lattice drop
        {'name': 'iteration_pile', 'kind': 'iteration', 'scene': 'pile', 'm': 6, 'layers': 5, 'n': 6},
        # a handful of settled bodies, the size that interactive users run
        {'name': 'iteration_small_pile', 'kind': 'iteration', 'scene': 'pile', 'm': 2, 'layers': 2, 'n': 5},
        # contact lists alone (a tool that inspects contacts frame by frame), uneven meshes
        {'name': 'constraints_pile', 'kind': 'constraints', 'scene': 'pile', 'm': 4, 'layers': 3, 'n': 7},
        # many uneven scenes together
        {'name': 'batch_64', 'kind': 'batch', 'scenes': 64},
        # the fallback and exact solver on a contact scene
        {'name': 'direct_pile', 'kind': 'direct', 'scene': 'pile', 'm': 3, 'layers': 3, 'n': 6},
        # the 2D path at its benchmark's size
        {'name': 'step_2d', 'kind': 'step2d', 'k': 16, 'n': 16},
        # the ADMM variant on two touching cubes of the configured mesh
        {'name': 'admm_two_cubes', 'kind': 'admm', 'n': 8},
        # the learned start: its training batch, and its evaluation over the largest scene
        {'name': 'train_8192', 'kind': 'train', 'rows': 8192},
        {'name': 'infer_176841', 'kind': 'infer', 'rows': 176841},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(['step', 'step', 'iteration', 'iteration', 'constraints', 'batch', 'direct', 'step2d', 'admm', 'train', 'infer'])
    layout = {'layout': rng.randint(1, 9999)}   # turns and offsets of the scene's bodies
    pile = {'scene': 'pile', 'm': rng.randint(1, 5), 'layers': rng.randint(2, 4), 'n': rng.randint(3, 7), **layout}
    bar = {'scene': 'bar', 'nx': _log_int(rng, 12, 250), 'ny': rng.randint(4, 18), 'nz': rng.randint(4, 18)}
    if kind == 'step':
        return {'kind': kind, **rng.choice([bar, {'scene': 'cubes', 'n': rng.randint(3, 9), **layout}])}
    if kind == 'iteration':
        return {'kind': kind, **rng.choice([bar, pile])}
    if kind == 'constraints':
        return {'kind': kind, **pile}
    if kind == 'batch':
        return {'kind': kind, 'scenes': _log_int(rng, 2, 60), **layout}
    if kind == 'direct':
        return {'kind': kind, **pile, 'm': rng.randint(1, 3), 'layers': rng.randint(1, 3), 'n': rng.randint(3, 6)}
    if kind == 'step2d':
        return {'kind': kind, 'k': rng.randint(2, 16), 'n': rng.randint(4, 18), **layout}
    if kind == 'admm':
        return {'kind': kind, 'n': rng.randint(3, 8), **layout}
    return {'kind': kind, 'rows': _log_int(rng, 100, 60000 if kind == 'train' else 170000)}


# ------------------------------------------------------------------------------------- scenes
def _pile(m, layers, n, layout, side=0.1):
    """Settled cubes: layers of m x m cubes of n hexes a side over a fixed ground box, each layer
    shifted by half a pitch, so that a cube rests on up to four below it, GAP contact distances
    away; every cube is turned a little about the vertical."""
    rng = np.random.default_rng(layout)
    base, tets = scenes.hex_grid(n, n, n, (side, side, side))
    pitch, lift = 1.25 * side, side + GAP * DHAT
    parts = []
    for b in range(layers):
        for a in range(m):
            for c in range(m):
                turn = scenes.rotation_matrix((0.0, 1.0, 0.0), rng.uniform(-0.26, 0.26))
                at = np.array([(a + 0.5 * (b % 2)) * pitch, GAP * DHAT + b * lift + side / 2, (c + 0.5 * (b % 2)) * pitch])
                parts.append(((base - side / 2) @ turn.T + at, tets))
    extent = (m + 1) * pitch
    ground, gt = scenes.hex_grid(1, 1, 1, (2 * extent, 0.1, 2 * extent))
    parts.append((ground + np.array([-0.75 * extent, -0.1, -0.75 * extent]), gt))
    return _scene('pile', parts, fixed_last=len(ground))


def _two_cubes_touching(n, layout, side=0.1):
    """Two cubes of n hexes a side, the lower one's bottom face fixed, GAP contact distances apart."""
    base, tets = scenes.hex_grid(n, n, n, (side, side, side))
    turn = scenes.rotation_matrix((0.0, 1.0, 0.0), np.random.default_rng(layout).uniform(-0.26, 0.26))
    up = (base - side / 2) @ turn.T + np.array([side / 2, 1.5 * side + GAP * DHAT, side / 2])
    sc = _scene('two_cubes', [(base, tets), (up, tets)], fixed_last=0)
    mask = np.zeros(len(sc.x), dtype=bool)
    mask[:len(base)] = base[:, 1] <= 1e-12
    return _fix(sc, mask)


def _scene(name, parts, fixed_last):
    offsets = np.cumsum([0] + [len(x) for x, _ in parts])
    x = np.concatenate([p for p, _ in parts])
    tets = np.concatenate([t + o for (_, t), o in zip(parts, offsets)]).astype(np.int32)
    points, edges, triangles = scenes.find_boundary(tets)
    sc = scenes.Scene(name, x, tets, np.zeros_like(x), points, edges, triangles, None, dhat=DHAT, dt=DT)
    mask = np.zeros(len(x), dtype=bool)
    if fixed_last:
        mask[-fixed_last:] = True
    return _fix(sc, mask)


def _fix(sc, mask):
    rest = sc.x.copy()
    sc.dirichlet = lambda t: (mask, rest)
    sc.dirichlet_groups = np.where(mask, 0, -1).astype(np.int32)
    sc.dirichlet_motion = scenes.motion_row()[None, :]
    return sc


def _column_2d(k, n, layout, side=0.1):
    """A column of k squares, GAP contact distances apart, over a fixed ground segment."""
    rng = np.random.default_rng(layout)
    base, tri = scenes.tri_grid(n, n, (side, side))
    parts = [base + np.array([rng.uniform(-0.1, 0.1) * side, GAP * DHAT + q * (side + GAP * DHAT)]) for q in range(k)]
    tris = np.concatenate([tri + q * len(base) for q in range(k)]).astype(np.int32)
    points, edges = scenes.find_boundary_2d(tris)
    free = k * len(base)
    x = np.concatenate(parts + [np.array([[-1.0, 0.0], [1.0, 0.0]])])
    points = np.concatenate([points, [free, free + 1]]).astype(np.int32)
    edges = np.concatenate([edges, [[free, free + 1]]]).astype(np.int32)
    mask = np.arange(len(x)) >= free
    rest = x.copy()
    return scenes.Scene2D('column_2d', x, tris, np.zeros_like(x), points, edges, lambda t: (mask, rest), dhat=DHAT, dt=DT)


def _make_scene(case):
    if case['scene'] == 'cubes':
        return scenes.two_cubes(n=case['n'], seed=case.get('layout', 0))
    if case['scene'] == 'bar':
        h = 0.0025
        return scenes.twisted_bar(nx=case['nx'], ny=case['ny'], nz=case['nz'], size=(case['nx'] * h, case['ny'] * h, case['nz'] * h))
    return _pile(case['m'], case['layers'], case['n'], case.get('layout', 0))


@lru_cache(maxsize=1)
def _object(key):
    """The simulation object that a program keeps, for a case's sizes."""
    case = dict(key)
    kind = case['kind']
    layout = case.get('layout', 0)
    if kind == 'batch':   # columns of 1 to 8 cubes
        return BatchNewtonIPC([_pile(1, k, n, 1000 * layout + q) for q, (k, n) in enumerate(_columns(case))], device=DEV, pcg_rtol=1e-12)
    if kind == 'step2d':
        return NewtonIPC2D(_column_2d(case['k'], case['n'], layout), device=DEV, pcg_rtol=1e-12)
    if kind == 'admm':
        return AdmmIPC(_two_cubes_touching(case['n'], layout), device=DEV)
    if kind == 'direct':
        return NewtonIPC(_make_scene(case), device=DEV, solver='direct')
    return NewtonIPC(_make_scene(case), device=DEV, **({'pcg_rtol': 1e-12} if kind == 'iteration' else {}))


def _columns(case):
    rng = np.random.default_rng(case.get('layout', 0))
    return [(int(rng.integers(1, 9)), int(rng.integers(3, 11))) for _ in range(case['scenes'])]


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != 'name'))


def _state_arrays(case, sim, seed):
    """Positions and velocities of the seed's state, on the host."""
    rng = np.random.default_rng(seed)
    if case['kind'] == 'batch':
        rest, fixed = np.concatenate([s.x for s in sim.scenes]), np.concatenate([s.dirichlet(0.0)[0] for s in sim.scenes])
    else:
        rest, fixed = sim.scene.x, sim.scene.dirichlet(0.0)[0]
    if case.get('scene') == 'bar':
        # the twist of the steps before, spread along the bar, and the velocity that goes with it
        half = np.abs(rest[:, 0]).max()
        rate = np.pi * rest[:, 0] / half * 0.5 * (1.0 + (rest[:, 0] / half) ** 2)
        ang = rate * (BAR_STEP - 1) * DT
        x = rest.copy()
        x[:, 1] = np.cos(ang) * rest[:, 1] - np.sin(ang) * rest[:, 2]
        x[:, 2] = np.sin(ang) * rest[:, 1] + np.cos(ang) * rest[:, 2]
        v = np.stack([np.zeros_like(rate), -rate * x[:, 2], rate * x[:, 1]], axis=1)
        x += rng.uniform(-2e-5, 2e-5, x.shape) * ~fixed[:, None]
        return x, v
    # vertices off the rest shape by up to a tenth of the contact distance, slow motion
    x = rest + rng.uniform(-0.1 * DHAT, 0.1 * DHAT, rest.shape) * ~fixed[:, None]
    v = rng.uniform(-0.01, 0.01, rest.shape) * ~fixed[:, None]
    if case.get('scene') == 'cubes':
        v = v + sim.scene.v
    return x, v


def _mlp_arrays(case, seed):
    """Features (one-ring offsets, velocity, last displacement, contact distance; 55 of 64 used),
    targets and parameters, on the GPU."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = case['rows']
    X = 0.3 * torch.randn((n, 64), generator=g, device=DEV)
    X[:, 54] = torch.rand(n, generator=g, device=DEV)
    X[:, 55:] = 0.0
    Y = torch.randn((n, 4), generator=g, device=DEV)
    Y[:, 3] = 0.0
    parts = []
    for rows, cols in ((128, 64), (128, 128), (128, 128), (4, 128)):
        parts.append(torch.randn(rows * cols, generator=g, device=DEV) * (2.0 / cols) ** 0.5)
        parts.append(0.1 * torch.randn(rows, generator=g, device=DEV))
    moments = 1e-3 * torch.randn(2, sum(p.numel() for p in parts), generator=g, device=DEV)
    return X.contiguous(), Y.contiguous(), torch.cat(parts), moments


def prepare(case, seed):
    if case['kind'] in ('train', 'infer'):
        X, Y, params, moments = _mlp_arrays(case, seed)
        model = WarmStartMLP(device=DEV, params=params)
        if case['kind'] == 'train':   # in mid-training: the optimiser has a history
            model.m.copy_(moments[0])
            model.v.copy_(moments[1] ** 2 + 1e-6)
            model.t = 1000
        return {'kind': case['kind'], 'model': model, 'X': X, 'Y': Y}
    sim = _object(_key(case))
    x, v = _state_arrays(case, sim, seed)
    return {'kind': case['kind'], 'sim': sim, 'frame': BAR_STEP if case.get('scene') == 'bar' else 0,
            'x': torch.tensor(x, device=DEV), 'v': torch.tensor(v, device=DEV)}


# ------------------------------------------------------------------------------------- passes
def run(state):
    kind = state['kind']
    if kind == 'train':
        m = state['model']
        loss = m.train_step(state['X'], state['Y'], lr=1e-3)
        return {'loss': loss, 'grads': m.grads, 'params': m.params}
    if kind == 'infer':
        return state['model'].forward(state['X'])
    return _RUN[kind](state['sim'], state['x'], state['v'], state['frame'])


def _step(sim, x, v, f):
    sim.set_state(x, v)
    its = sim.step(f)
    return {'x': sim.x, 'v': sim.v, 'iterations': its}


def _start(sim, x, v, f):
    sim.set_state(x, v)
    sim.compute_xn_and_xTilde()
    sim.move_nodes(f * DT)


def _iteration(sim, x, v, f):
    _start(sim, x, v, f)
    counts = list(sim.find_constraints())
    sim.compute_hessian_and_gradient()
    sim.solve_system(f * DT)
    out = {'counts': counts, 'residual': sim.output_residual(), 'E0': sim.compute_energy()}
    sim.save_xPrev()
    out['alpha'] = sim.compute_intersection_free_step_size()
    sim.apply_sol(out['alpha'])
    out['hit'] = sim.check_collision()
    out['counts_trial'] = list(sim.find_constraints())
    out['E'] = sim.compute_energy()
    out['direction'], out['x'] = sim.data_sol, sim.x
    return out


def _constraints(sim, x, v, f):
    sim.set_state(x, v)
    counts = list(sim.find_constraints())
    # into the caller's own buffers, which do not change their size with the state
    out = [np.zeros((2 * len(sim.scene.boundary_points) + 16, w), np.int32) for w in (2, 3, 4, 4, 4, 4, 4)]
    for to, rows in zip(out, sim.constraints()):
        to[:len(rows)] = rows
    return {'counts': counts, 'rows': out}


def _direct(sim, x, v, f):
    _start(sim, x, v, f)
    sim.find_constraints()
    sim.compute_hessian_and_gradient()
    sim.solve_system(f * DT)
    return {'direction': sim.data_sol, 'residual': sim.output_residual()}


def _batch(sim, x, v, f):
    sim.x.copy_(x)
    sim.v.copy_(v)
    sim.compute_xn_and_xTilde()
    sim.move_nodes(0.0)
    counts = list(sim.find_constraints())
    sim.compute_hessian_and_gradient()
    sim.solve_system(0.0)
    residual = sim.output_residual()
    sim.compute_energy(sim.E0)
    sim.save_xPrev()
    sim.compute_intersection_free_step_size()
    sim.apply_sol()
    hit = sim.check_collision()
    trial = list(sim.find_constraints())
    sim.compute_energy()
    return {'counts': counts, 'counts_trial': trial, 'residual': residual, 'hit': hit, 'E0': sim.E0, 'E': sim.E, 'alpha': sim.alpha,
            'direction': sim.data_sol, 'x': sim.x}


def _admm(sim, x, v, f):
    sim.set_state(x, v)
    sim.admm_initial_guess()
    sim.admm_iteration(0, 0)
    sim.admm_iteration(0, 1)
    # the rows' variables into buffers that do not change their size with the state
    cap = 2 * len(sim.scene.boundary_points) + 16
    fixed = lambda a: torch.nn.functional.pad(a, (0, 0) * (a.dim() - 1) + (0, cap - len(a)))  # noqa: E731
    return {'x': sim.x, 'z': sim.z, 'u': sim.u, 'rows': fixed(sim.rows_all), 'y': fixed(sim.y), 'r': fixed(sim.r), 'Q': fixed(sim.Q)}


_RUN = {'step': _step, 'iteration': _iteration, 'constraints': _constraints, 'direct': _direct, 'batch': _batch, 'step2d': _step,
        'admm': _admm}


# ------------------------------------------------------------------------------------- work
def _sizes(case):
    """(vertices, tets or triangles) of a case's scenes."""
    kind = case['kind']
    if kind == 'batch':
        return sum(k * (n + 1) ** 3 + 8 for k, n in _columns(case)), sum(6 * k * n ** 3 + 6 for k, n in _columns(case))
    if kind == 'step2d':
        return case['k'] * (case['n'] + 1) ** 2 + 2, 2 * case['k'] * case['n'] ** 2
    if kind == 'admm' or case['scene'] == 'cubes':
        return 2 * (case['n'] + 1) ** 3, 12 * case['n'] ** 3
    if case['scene'] == 'bar':
        return (case['nx'] + 1) * (case['ny'] + 1) * (case['nz'] + 1), 6 * case['nx'] * case['ny'] * case['nz']
    cubes = case['m'] ** 2 * case['layers']
    return cubes * (case['n'] + 1) ** 3 + 8, 6 * cubes * case['n'] ** 3 + 6


def work(case):
    """The state and the mesh read once, the state written once; for a solve also the element
    Hessians' arithmetic (about 1,800 operations a tet, 300 a triangle) and one product with the
    system (18 operations a 3x3 block, about 15 blocks a vertex), since how often a solver has to
    apply it is its own affair; for the network its products."""
    kind = case['kind']
    if kind in ('train', 'infer'):
        n, weights = case['rows'], 128 * 64 + 2 * 128 * 128 + 4 * 128
        if kind == 'train':
            return {'bytes': 4 * (n * 68 + 8 * 41860), 'flops': 2 * n * (3 * weights - 128 * 64)}
        return {'bytes': 4 * (n * 68 + 41860), 'flops': 2 * n * weights}
    nv, nt = _sizes(case)
    if kind == 'step2d':
        return {'bytes': 2 * 32 * nv + 68 * nt, 'flops': 300 * nt + 8 * 7 * nv}
    if kind == 'constraints':
        return {'bytes': 24 * nv, 'flops': 24 * nv}
    return {'bytes': 2 * 48 * nv + 112 * nt, 'flops': 1800 * nt + 18 * 15 * nv}


# ------------------------------------------------------------------------------------- 64 bits
def exact(case, seed):
    if case['kind'] == 'infer':
        X, _, params, _ = _mlp_arrays(case, seed)
        return _network(X.double(), [p.double() for p in _split(params)])
    if case['kind'] == 'train':
        return _exact_train(case, seed)
    if case['kind'] == 'iteration' and case['scene'] == 'bar' and _sizes(case)[1] <= 200000:
        return _exact_bar(case, seed)
    return None


def _split(flat):
    parts, at = [], 0
    for rows, cols in ((128, 64), (128, 128), (128, 128), (4, 128)):
        parts.append(flat[at:at + rows * cols].view(rows, cols))
        parts.append(flat[at + rows * cols:at + rows * cols + rows])
        at += rows * cols + rows
    return parts


def _network(h, parts):
    for k in range(3):
        h = torch.nn.functional.gelu(h @ parts[2 * k].T + parts[2 * k + 1])
    return h @ parts[6].T + parts[7]


def _exact_train(case, seed):
    X, Y, params, moments = _mlp_arrays(case, seed)
    flat = params.double().requires_grad_(True)
    d = (_network(X.double(), _split(flat)) - Y.double())[:, :3]
    loss = (d * d).mean()
    loss.backward()
    g = flat.grad
    # the optimiser's constants are single-precision numbers: lr, its two decay rates and epsilon
    lr, b1, b2, eps = (float(np.float32(c)) for c in (1e-3, 0.9, 0.999, 1e-8))
    m = b1 * moments[0].double() + (1 - b1) * g
    v = b2 * (moments[1] ** 2 + 1e-6).double() + (1 - b2) * g * g
    new = flat.detach() - lr * (m / (1 - b1 ** 1001)) / ((v / (1 - b2 ** 1001)).sqrt() + eps)
    return {'loss': loss.detach().reshape(1), 'grads': g, 'params': new}


def _exact_bar(case, seed):
    """The first energy, the Newton direction and its largest entry of a bar's iteration: element
    matrices from numpy's singular values, conjugate gradients on them to 1e-14 in torch."""
    sc = _make_scene(case)

    class _Scene:   # what _state_arrays reads
        scene = sc
    x, v = _state_arrays(case, _Scene, seed)
    fixed, target = sc.dirichlet(BAR_STEP * DT)
    xt = x + DT * v
    xt[:, 1] += DT * DT * sc.gravity
    x[fixed] = target[fixed]
    xt[fixed] = target[fixed]
    t = sc.tets
    edges = lambda p: np.stack([p[t[:, k + 1]] - p[t[:, 0]] for k in range(3)], axis=2)  # noqa: E731
    Dm = edges(sc.x)
    vol = np.linalg.det(Dm) / 6.0
    mass = np.zeros(len(x))
    np.add.at(mass, t.ravel(), np.repeat(vol * sc.rho / 4.0, 4))
    IB = np.linalg.inv(Dm)
    mu, la = sc.E / (2 * (1 + sc.nu)), sc.E * sc.nu / ((1 + sc.nu) * (1 - 2 * sc.nu))
    F = edges(x) @ IB
    U, s, Vt = np.linalg.svd(F)
    for Q in (U, np.swapaxes(Vt, 1, 2)):   # rotations; F keeps its orientation, so s stays positive
        Q[:, :, 2] *= np.sign(np.linalg.det(Q))[:, None]
    lp = np.log(s.prod(axis=1))
    w = DT * DT * vol
    energy = 0.5 * (mass * ((x - xt) ** 2).sum(axis=1)).sum() + (w * (mu / 2 * ((s * s).sum(axis=1) - 3) - (mu - la / 2 * lp) * lp)).sum()
    # the stress and its projected derivative in the basis u_a v_b^T
    gs = mu * (s - 1 / s) + la * lp[:, None] / s
    P = (U * gs[:, None, :]) @ Vt
    M = np.zeros((len(t), 3, 3, 3, 3))
    H = la / (s[:, :, None] * s[:, None, :])
    for i in range(3):
        H[:, i, i] = mu * (1 + 1 / s[:, i] ** 2) - la / s[:, i] ** 2 * (lp - 1)
    e, q = np.linalg.eigh(H)
    H = np.where((e[:, :1, None] < 0), (q * np.maximum(e, 0)[:, None, :]) @ np.swapaxes(q, 1, 2), H)
    for i in range(3):
        for j in range(3):
            M[:, i, i, j, j] = H[:, i, j]
    for i, j in ((0, 1), (1, 2), (2, 0)):
        left = (mu + (mu - la * lp) / (s[:, i] * s[:, j])) / 2
        right = (gs[:, i] + gs[:, j]) / (2 * np.maximum(s[:, i] + s[:, j], 1e-6))
        # the reference's 2x2 projection: where right < 0 both entries become (left - right)^2 / (2 left)
        on, off = np.where(right < 0, 0.5 * (left - right) ** 2 / left, left + right), np.where(right < 0, 0.5 * (left - right) ** 2 / left, left - right)
        M[:, i, j, i, j], M[:, j, i, j, i], M[:, i, j, j, i], M[:, j, i, i, j] = on, on, off, off
    B = np.concatenate([-IB.sum(axis=1, keepdims=True), IB], axis=1)     # shape gradients, vertex by vertex
    f64 = lambda a: torch.tensor(a, dtype=torch.float64, device=DEV)  # noqa: E731
    U_, z, M_ = f64(U), f64(np.einsum('eva,eba->evb', B, Vt)), f64(M)    # z: in the basis v_b
    K = torch.einsum('eabcd,evb,ewd->evawc', M_, z, z)
    K = torch.einsum('eia,evawc,ejc->eviwj', U_, K, U_) * f64(w)[:, None, None, None, None]
    K = K.reshape(len(t), 12, 12).contiguous()
    T, mass_, free = torch.tensor(t.astype(np.int64), device=DEV), f64(mass), f64((~fixed).astype(float))[:, None]
    force = torch.zeros((len(x), 3), dtype=torch.float64, device=DEV)
    force.index_add_(0, T.reshape(-1), torch.einsum('eij,evj->evi', f64(P), f64(B)).mul(f64(w)[:, None, None]).reshape(-1, 3))
    rhs = -(mass_[:, None] * f64(x - xt) + force) * free

    def apply(p):
        y = mass_[:, None] * p
        y.index_add_(0, T.reshape(-1), torch.bmm(K, p[T].reshape(-1, 12, 1)).reshape(-1, 3))
        return y * free
    D = mass_[:, None, None] * torch.eye(3, dtype=torch.float64, device=DEV)
    for k in range(4):
        D.index_add_(0, T[:, k], K[:, 3 * k:3 * k + 3, 3 * k:3 * k + 3].contiguous())
    inv = torch.linalg.inv(D)
    sol, r = torch.zeros_like(rhs), rhs.clone()
    p = z0 = torch.einsum('vij,vj->vi', inv, r)
    rz, stop = (r * z0).sum(), 1e-28 * float((rhs * rhs).sum())
    for it in range(20000):
        Ap = apply(p)
        step = rz / (p * Ap).sum()
        sol, r = sol + step * p, r - step * Ap
        if it % 50 == 49 and float((r * r).sum()) <= stop:
            break
        z0 = torch.einsum('vij,vj->vi', inv, r)
        rz, old = (r * z0).sum(), rz
        p = z0 + (rz / old) * p
    return {'counts': [None] * 7, 'residual': float(sol.abs().max()), 'E0': float(energy), 'alpha': None, 'hit': None,
            'counts_trial': [None] * 7, 'E': None, 'direction': sol, 'x': None}
