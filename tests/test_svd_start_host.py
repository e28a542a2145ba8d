"""The 3x3 SVD from its FP32 start, compiled for the host, where the start can go wrong: equal and nearly
equal singular values, condition numbers to 1e6, reflections, and entries outside FP32's range.

Bar: Jacobi on the columns leaves each singular value within a few units of its own rounding and the
factors orthonormal; U S V^T reproduces F to 64 eps of its norm, orthonormality to 64 eps."""
import ctypes

import numpy as np
import pytest

from tests.test_device_math_host import P, hc  # noqa: F401

EPS = np.finfo(float).eps


@pytest.mark.parametrize('scale', [1.0, 1e-30, 1e30, 1e-60])
@pytest.mark.parametrize('s', [(1, 1, 1), (1.1, 1.1, 0.9), (1, 1 - 1e-8, 1 - 2e-8), (1, 0.5, 1e-6), (1.2, 0.9, -0.3), (2, 1e-3, 1e-3)])
def test_svd(hc, s, scale):  # noqa: F811
    rng = np.random.default_rng(3)
    N = 200
    U0, V0 = (np.linalg.qr(rng.normal(size=(N, 3, 3)))[0] for _ in range(2))
    for Q in (U0, V0):
        Q *= np.sign(np.linalg.det(Q))[:, None, None]
    F = np.ascontiguousarray(scale * np.einsum('nij,j,nkj->nik', U0, np.array(s, float), V0))
    U, sv, V = np.zeros((N, 3, 3)), np.zeros((N, 3)), np.zeros((N, 3, 3))
    hc.hc_svd3(N, P(F), P(U), P(sv), P(V))
    n = np.abs(F).max(axis=(1, 2))
    assert (np.abs(np.einsum('nij,nj,nkj->nik', U, sv, V) - F).max(axis=(1, 2)) <= 64 * EPS * n).all()
    for Q in (U, V):
        assert np.abs(np.einsum('nij,nik->njk', Q, Q) - np.eye(3)).max() <= 64 * EPS
        np.testing.assert_allclose(np.linalg.det(Q), 1, atol=1e-14)
    want = np.array(sorted(np.abs(s), reverse=True)) * scale
    assert (np.abs(np.abs(sv) - want) <= 64 * EPS * want[0]).all()
    assert (np.sign(sv[:, 2]) == np.sign(np.prod(s))).all()
