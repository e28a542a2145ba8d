"""The step filter's sign test over pairs: a pair that it leaves out has no impact in the oracle's interval test.  Near pairs in
general position, slow and fast, with and without a common translation, small and large."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import oracle as O

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, 'native', 'ccd_apart_host.cpp')
OUT = os.path.join(HERE, 'native', '_build', 'ccd_apart_host.so')
P = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731


@pytest.fixture(scope='module')
def hc():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + f'.{os.getpid()}'
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-fPIC', '-shared', SRC, '-o', tmp])
    os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


@pytest.mark.parametrize('speed', [0.05, 0.5, 3.0])
@pytest.mark.parametrize('size', [1e-3, 1.0])
@pytest.mark.parametrize('drift', [0.0, 2.0])
@pytest.mark.parametrize('kind', [0, 1])
def test_left_out_pairs_do_not_meet(hc, kind, drift, size, speed):
    rng = np.random.default_rng(int(100 * speed + 10 * drift + kind))
    N = 20000
    x = rng.uniform(-0.5, 0.5, (N, 4, 3))
    if kind == 0:
        x[:, 0] = x[:, 1:].mean(1) + 0.3 * rng.normal(size=(N, 3))
    else:
        x[:, 2:] += (x[:, :2].mean(1) - x[:, 2:].mean(1) + 0.3 * rng.normal(size=(N, 3)))[:, None]
    p = speed * rng.uniform(-1, 1, (N, 4, 3)) + drift * rng.uniform(-1, 1, (N, 1, 3))
    x, p = np.ascontiguousarray(size * x), np.ascontiguousarray(size * p)
    apart = np.zeros(N, np.int32)
    hc.hc_apart(kind, N, P(x), P(p), ctypes.c_double(0.2), P(apart))
    toc = O.ccd(kind, x, p, 0.2)
    assert (toc[apart != 0] == 1.0).all()
    assert apart.any()   # 99% of the slow pairs, a quarter of the fastest
