"""Symmetric eigen-solver (host build of eig.cuh) on matrices of order one whose last row is coupled to the others by
subnormal numbers only, whose reciprocal is infinite.

Bar: the method is backward stable, so eigenvalues and the rebuilt matrix are within some n^2 eps |A| of the exact ones:
81 x 2.2e-16 x 6 (the largest norm here) is 1.1e-13; 1e-12."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, 'native', 'math_host.cpp')
OUT = os.path.join(HERE, 'native', '_build', 'eig_small_rows_host.so')
P = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731


@pytest.fixture(scope='module')
def hc():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + f'.{os.getpid()}'
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-fPIC', '-shared', SRC, '-o', tmp])
    os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


@pytest.mark.parametrize('size', [1e-307, 1e-308, 1e-310, 1e-316, 5e-324])
@pytest.mark.parametrize('n', [3, 6, 9])
def test_subnormal_row(hc, n, size):
    rng = np.random.default_rng(n)
    N = 20
    A = rng.uniform(-1, 1, (N, n, n))
    A = (A + A.transpose(0, 2, 1)) / 2
    A[:, -1, :-1] = A[:, :-1, -1] = size * np.sign(rng.uniform(-1, 1, (N, n - 1)))
    A = np.ascontiguousarray(A)
    w, V = np.zeros((N, n)), np.zeros((N, n, n))
    hc.hc_sym_eig(N, n, P(A), P(w), P(V))
    np.testing.assert_allclose(w, np.linalg.eigvalsh(A), rtol=0, atol=1e-12)
    np.testing.assert_allclose(np.einsum('bij,bj,bkj->bik', V, w, V), A, rtol=0, atol=1e-12)
