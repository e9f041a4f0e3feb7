"""Singular values in pairs 1e-10 apart (relative): their Ritz vectors leave the
twisted factorisations for the QR kernels.  The Krylov space is as large as the
matrix, so every triplet is exact to rounding: 64 m eps sigma_1, as in
test_bidiag.py, and the vectors of a pair are orthonormal to the same level."""
import numpy as np
import pytest

import propack_gb300 as pg

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


@pytest.mark.parametrize("irl", [False, True])
@pytest.mark.parametrize("m,n", [(400, 300), (300, 400), (60, 60)])
def test_pairs(m, n, irl):
    r, k = min(m, n), 20
    rng = np.random.default_rng(m)
    s = np.repeat(np.linspace(2.0, 1.0, r // 2), 2)
    s[1::2] *= 1.0 - 3e-10
    q1 = np.linalg.qr(rng.standard_normal((m, r)))[0]
    q2 = np.linalg.qr(rng.standard_normal((n, r)))[0]
    A = (q1 * s) @ q2.T
    u, sg, vt, _ = pg.svdp(A, k, irl_mode=irl, kmax=r, tol=1e-10, delta=0.0, rng=np.random.default_rng(0))
    tol = (1e-10 if irl else 0.0) + 64 * max(m, n) * EPS
    assert np.max(np.abs(sg - s[:k])) <= tol * s[0]
    assert np.max(np.linalg.norm(A @ vt.T - u * sg, axis=0)) <= tol * s[0]
    assert np.max(np.linalg.norm(A.T @ u - vt.T * sg, axis=0)) <= tol * s[0]
    assert np.max(np.abs(u.T @ u - np.eye(k))) <= 64 * max(m, n) * EPS
    assert np.max(np.abs(vt @ vt.T - np.eye(k))) <= 64 * max(m, n) * EPS
