"""The reciprocal of pivots against division: within one ulp over all magnitudes, with the division itself outside the range
of its FP32 start; signs, zero, infinities and NaN as the division gives them."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, 'native', 'reciprocal_host.cpp')
OUT = os.path.join(HERE, 'native', '_build', 'reciprocal_host.so')


@pytest.fixture(scope='module')
def recip():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + f'.{os.getpid()}'
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-fPIC', '-shared', SRC, '-o', tmp])
    os.replace(tmp, OUT)
    lib = ctypes.CDLL(OUT)

    def f(d):
        d = np.ascontiguousarray(d, dtype=np.float64)
        r = np.empty_like(d)
        lib.hc_reciprocal(len(d), d.ctypes.data_as(ctypes.c_void_p), r.ctypes.data_as(ctypes.c_void_p))
        return r
    return f


def test_within_an_ulp(recip):
    rng = np.random.default_rng(0)
    d = rng.uniform(1, 2, 400000) * 2.0 ** rng.integers(-99, 99, 400000)
    d = np.concatenate([d, 2.0 ** np.arange(-1000.0, 1000.0), 1 + 2.0 ** -np.arange(1.0, 53.0), 2 - 2.0 ** -np.arange(1.0, 53.0)])
    w = 1.0 / d
    assert (np.abs(recip(d) - w) <= np.spacing(w)).all()


def test_special_values(recip):
    d = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, -3e-7, 5e-324, 1e-30, 1e30, 1e-31, 1e31, 1e300, 1e-300])
    with np.errstate(divide='ignore', over='ignore'):
        w = 1.0 / d
    r = recip(d)
    special = ~((d >= 1e-30) & (d <= 1e30))
    np.testing.assert_array_equal(r[special], w[special])
    assert (np.abs(r[~special] - w[~special]) <= np.spacing(w[~special])).all()
