"""Contribution lists of an aggregated pattern against a lexicographic sort (numpy): order by coarse row, coarse
column, source position, exactly; sizes that shrink and grow between calls on the same buffers, empty
patterns, Dirichlet rows and columns left out."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, 'native', 'mg_pattern_host.cpp')
OUT = os.path.join(HERE, 'native', '_build', 'mg_pattern_host.so')


@pytest.fixture(scope='module')
def hc():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + f'.{os.getpid()}'
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-fPIC', '-shared', SRC, '-o', tmp])
    os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


@pytest.mark.parametrize('fix', [False, True])
def test_lists(hc, fix):
    rng = np.random.default_rng(fix)
    P = lambda a: None if a is None else a.ctypes.data_as(ctypes.c_void_p)
    for n, nc, deg in [(500, 40, 12), (7, 3, 4), (1, 1, 1), (2000, 300, 25), (30, 30, 0), (900, 5, 9)]:
        rows = [np.unique(rng.integers(0, n, rng.integers(0, deg + 1))) if deg else np.zeros(0, int) for _ in range(n)]
        rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
        ci = np.concatenate(rows).astype(np.int32)
        agg = rng.integers(0, nc, n).astype(np.int32)
        fixed = (rng.random(n) < 0.2).astype(np.uint8) if fix else None
        i = np.repeat(np.arange(n), np.diff(rp))
        k = np.arange(len(ci))
        if fix:
            keep = ~(fixed[i] | fixed[ci]).astype(bool)
            i, k = i[keep], k[keep]
        I, J = agg[i], agg[ci[k]]
        o = np.lexsort((k, J, I))
        i, k, I, J = i[o], k[o], I[o], J[o]
        first = np.flatnonzero(np.concatenate([[True], (np.diff(I) != 0) | (np.diff(J) != 0)])) if len(k) else np.zeros(0, int)
        b = [np.zeros(max(len(ci), 1) + 2, np.int32) for _ in range(5)]
        orp, ns = np.zeros(nc + 1, np.int32), ctypes.c_int()
        nnz = hc.hc_pattern(n, P(rp), P(ci), P(agg), nc, P(fixed), P(orp), *[P(x) for x in b], ctypes.byref(ns))
        assert nnz == len(first) and ns.value == len(k)
        np.testing.assert_array_equal(orp, np.concatenate([[0], np.cumsum(np.bincount(I[first], minlength=nc))]))
        np.testing.assert_array_equal(b[0][:nnz], J[first])
        np.testing.assert_array_equal(b[1][:nnz + 1], np.concatenate([first, [len(k)]]) if len(k) else [0])
        for got, want in zip(b[2:], (k, i, ci[k])):
            np.testing.assert_array_equal(got[:len(k)], want)
