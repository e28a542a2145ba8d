"""Root isolation of the step filter in the Bernstein basis, compiled for the host, on polynomials with known
roots: inside, outside and near the ends of [0, 1], pairs from far apart to almost double, complex pairs.

Bars.  Roots given up (count -1) only for polynomials with a Bernstein coefficient near zero: a root within
1e-9 of a halving point or end, or pairs closer than the deepest halving separates (2^-10, at a root's
neighbourhood of up to a few segments).  A returned root of a polynomial whose largest coefficient is 1 and whose
slope there is s is off by at most 1e-14 / |s| (the coefficients' rounding in construction and Horner's)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, 'native', 'ccd_roots_host.cpp')
OUT = os.path.join(HERE, 'native', '_build', 'ccd_roots_host.so')


@pytest.fixture(scope='module')
def hc():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + f'.{os.getpid()}'
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-ffp-contract=off', '-fPIC', '-shared', SRC, '-o', tmp])
    os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


def run(hc, n, op):
    P = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    N = len(op)
    a, b = np.zeros((N, 8)), np.zeros((N, 8))
    na, nb, ep, en = (np.zeros(N, np.int32) for _ in range(4))
    hc.hc_roots(n, N, P(np.ascontiguousarray(op)), P(a), P(na), P(b), P(nb), P(ep), P(en))
    return a, na, b, nb, ep, en


def polynomials(n, N, gap, rng):
    """[N, n+1] with n_in roots in (0, 1), two of them `gap` apart, the others outside or complex."""
    op, inside = [], []
    for _ in range(N):
        k = rng.integers(0, n + 1)
        r = list(rng.uniform(0.02, 0.98, k))
        if k >= 2:
            r[1] = min(r[0] + gap, 0.99)
        rest = n - k
        c = []
        while rest:
            if rest >= 2 and rng.random() < 0.5:
                z = complex(rng.uniform(-1, 2), rng.uniform(0.3, 1))
                c += [z, z.conjugate()]
                rest -= 2
            else:
                c.append(rng.uniform(1.05, 3) if rng.random() < 0.5 else rng.uniform(-3, -0.05))
                rest -= 1
        q = np.real(np.poly(r + c)) * rng.choice([-1, 1])
        op.append(q / np.abs(q).max())
        inside.append(sorted(r))
    return np.array(op), inside


@pytest.mark.parametrize('gap', [0.3, 0.03, 3e-3])
@pytest.mark.parametrize('n', [3, 4, 6])
def test_known_roots(hc, n, gap):
    op, inside = polynomials(n, 400, gap, np.random.default_rng(n))
    a, na, b, nb, ep, en = run(hc, n, op)
    assert (na >= 0).mean() > 0.8 if gap >= 0.03 else (na >= 0).mean() > 0.3
    for c in range(len(op)):
        if na[c] < 0:
            continue
        slope = np.polyval(np.polyder(op[c]), inside[c])
        if len(inside[c]) and np.abs(slope).min() < 1e-6:
            continue   # nearly double: the construction's rounding decides
        assert na[c] == len(inside[c]), c
        got = a[c, :na[c]]
        assert (np.diff(got) > 0).all()
        assert (np.abs(got - inside[c]) <= 1e-14 / np.abs(slope) + 1e-15).all(), (c, got, inside[c])
        if nb[c] == na[c]:
            assert (np.abs(got - b[c, :nb[c]]) <= 1e-14 / np.abs(slope) + 1e-15).all()


@pytest.mark.parametrize('n', [3, 4, 6])
def test_sign_filter_is_never_wrong(hc, n):
    op, _ = polynomials(n, 400, 0.1, np.random.default_rng(10 + n))
    scale = 10.0 ** np.random.default_rng(n).uniform(-9, 9, (len(op), 1))
    t = np.linspace(0, 1, 501)
    _, _, _, _, ep, en = run(hc, n, op * scale)
    v = np.array([np.polyval(q, t) for q in op])
    assert ep.sum() > 10 and en.sum() > 10
    assert (v[ep == 1] < 0).all() and (v[en == 1] > 0).all()


def test_degenerate(hc):
    """Zero, with a zero coefficient in the basis, NaN: nothing is decided."""
    op = np.array([[0, 0, 0, 0], [1, 0, 0, 0], [1, -1, 0, 0], [np.nan, 1, 1, 1]], float)
    _, na, _, _, ep, en = run(hc, 3, op)
    assert (na == -1).all() and not ep.any() and not en.any()
