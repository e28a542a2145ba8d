"""The order of posts, polls, clears and fences in the 2D PCG's slot exchange, on the CPU: three CTAs under a model of
relaxed accesses and fences, over seeded schedules.  The order in use reads no other epoch's value and no row
that is not the one stored before the exchange; orders that lack one of its parts are caught doing so."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, 'native', 'slot_order_host.cpp')
OUT = os.path.join(HERE, 'native', '_build', 'slot_order_host.so')


@pytest.fixture(scope='module')
def hc():
    os.makedirs(os.path.dirname(OUT), exist_ok=True)
    tmp = OUT + f'.{os.getpid()}'
    subprocess.check_call(['g++', '-O2', '-std=c++17', '-fPIC', '-shared', SRC, '-o', tmp])
    os.replace(tmp, OUT)
    return ctypes.CDLL(OUT)


def test_order_in_use(hc):
    assert hc.hc_slot_order(0, 4000) == 0


@pytest.mark.parametrize('order', [1, 2, 3])
def test_wrong_orders_are_caught(hc, order):
    assert hc.hc_slot_order(order, 4000) != 0
