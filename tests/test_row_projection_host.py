"""Projected Hessians of the unmollified constraint rows (host build of barrier.cuh): no negative eigenvalue beyond rounding,
over gaps from a tenth to 1e-8 of the geometry's size, up to the barrier's edge, and slivers.

Bar: an entry is a sum of at most nine products of up to four factors, some 40 roundings, and a row of the 12 x 12 matrix
adds up twelve of them: the lowest eigenvalue is above -480 eps of the largest; 500 eps."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, 'native', 'math_host.cpp')
OUT = os.path.join(HERE, 'native', '_build', 'row_projection_host.so')
P = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731


@pytest.fixture(scope='module')
def hc():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + f'.{os.getpid()}'
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-fPIC', '-shared', SRC, '-o', tmp])
    os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


def _unit(a):
    return a / np.linalg.norm(a, axis=-1, keepdims=True)


def _rows(t, N, gap, aspect, rng):
    o = rng.uniform(-0.5, 0.5, (N, 3))
    e1 = _unit(rng.normal(size=(N, 3)))
    b = _unit(np.cross(e1, rng.normal(size=(N, 3))))
    n = np.cross(e1, b)
    e2 = aspect * rng.uniform(0.3, 1, (N, 1)) * b + rng.uniform(-0.3, 0.3, (N, 1)) * e1
    u, v = rng.uniform(0.05, 0.95, (2, N, 1))
    s = gap * n
    if t == 0:
        X = [o, o + s, o, o]
    elif t == 1:
        X = [o + u * e1 + s, o, o + e1, o]
    elif t == 2:
        X = [o + u * e1 + v * (1 - u) * e2 + s, o, o + e1, o + e2]
    else:
        X = [o, o + e1, o + u * e1 + s - v * e2, o + u * e1 + s + (1 - v) * e2]
    return np.stack(X, axis=1)


@pytest.mark.parametrize('edge', [0.5, 0.99, 1 - 1e-9])
@pytest.mark.parametrize('gap,aspect', [(1e-1, 1.0), (1e-1, 1e-3), (1e-3, 1.0), (1e-3, 1e-3), (1e-6, 1.0), (1e-8, 1.0)])
@pytest.mark.parametrize('t', range(4))
def test_lowest_eigenvalue(hc, t, gap, aspect, edge):
    N, nv = 200, (2, 3, 4, 4)[t]
    X = _rows(t, N, gap, aspect, np.random.default_rng(t))
    rows = np.arange(4 * N, dtype=np.int32).reshape(N, 4)
    E, g, H = np.zeros(N), np.zeros((N, 12)), np.zeros((N, 144))
    hc.hc_barrier_rows(t, N, P(rows), P(X), P(X), ctypes.c_double((gap / edge) ** 2), ctypes.c_double(1e4), P(E), P(g), P(H))
    n = 3 * nv
    H = H[:, :n * n].reshape(N, n, n)
    assert np.isfinite(H).all()
    w = np.linalg.eigvalsh((H + H.transpose(0, 2, 1)) / 2)
    inside = w[:, -1] > 0   # rounding puts some distances at the edge outside
    assert inside.sum() > N // 4
    assert (w[inside, 0] >= -500 * 2.0 ** -53 * 2 * w[inside, -1]).all(), (w[:, 0] / w[:, -1]).min()
