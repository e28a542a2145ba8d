"""The broad phase's kept buffers when an allocation fails: no capacity counts that a buffer does not hold, and the next call
gets what it asks for."""
import ctypes
import os
import subprocess

import pytest

from fastipc_gb300.build import nvcc

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, 'native', 'grow_buffers_host.cpp')
OUT = os.path.join(HERE, 'native', '_build', 'grow_buffers_host.so')


@pytest.fixture(scope='module')
def hc():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + f'.{os.getpid()}'
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), 'include')
    subprocess.check_call(['g++', '-O1', '-std=c++17', '-fPIC', '-shared', '-Wl,-Bsymbolic', '-I', include, SRC, '-o', tmp])
    os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


@pytest.mark.parametrize('fail', range(4))
def test_tables(hc, fail):
    assert hc.hc_grid_after_failure(fail) == 0


@pytest.mark.parametrize('fail', range(3))
def test_rows(hc, fail):
    assert hc.hc_rows_after_failure(fail) == 0
