"""The small bidiagonal kernels (analysis and Ritz pairs) at the edges of
their warps and rescaling blocks: Lanczos runs to the full dimension of small
dense matrices, so that every bidiagonal value and vector counts.

Tolerances: every value and residual comes from O(n) roundings of numbers at
most sigma_1 (Lanczos with full reorthogonalisation, the bidiagonal SVD by
bisection to 2 eps, products of n terms), so 64 n eps sigma_1 bounds them.
"""
import numpy as np
import pytest

import propack_gb300 as pg

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _matrix(m, n, decay, rng):
    k = min(m, n)
    q1, _ = np.linalg.qr(rng.standard_normal((m, k)))
    q2, _ = np.linalg.qr(rng.standard_normal((n, k)))
    return (q1 * decay ** np.arange(k)) @ q2.T


@pytest.mark.parametrize("n", [1, 2, 3, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 130])
@pytest.mark.parametrize("shape", ["tall", "wide", "square"])
def test_full_dimension_values_and_vectors(n, shape):
    rng = np.random.default_rng(1000 * n)
    m = n + 7 if shape == "tall" else n
    A = _matrix(m, n, 0.9 if n < 60 else 0.97, rng)
    A = A.T.copy() if shape == "wide" else A
    u, s, vt, bnd = pg.svdp(A, n, irl_mode=False, kmax=n + 1, tol=1e-13, delta=0.0, rng=np.random.default_rng(0))
    ref = np.linalg.svd(A, compute_uv=False)
    tol = 64 * max(A.shape) * EPS * ref[0]
    assert np.max(np.abs(s - ref[:n])) <= tol
    assert np.max(np.abs(A @ vt.T - u * s)) <= tol
    assert np.max(np.abs(A.T @ u - vt.T * s)) <= tol
    assert np.max(np.abs(u.T @ u - np.eye(n))) <= 64 * max(A.shape) * EPS / (ref[n - 1] / ref[0])


@pytest.mark.parametrize("k,kmax", [(1, 2), (2, 5), (4, 33), (8, 64), (16, 65), (30, 150)])
def test_restarted_values_by_dimension(k, kmax):
    rng = np.random.default_rng(k)
    A = _matrix(400, 300, 0.93, rng)
    u, s, vt, bnd = pg.svdp(A, k, kmax=kmax, tol=1e-13, delta=0.0, rng=np.random.default_rng(0))
    ref = np.linalg.svd(A, compute_uv=False)
    tol = 64 * 400 * EPS * ref[0]
    assert np.max(np.abs(s - ref[:k])) <= tol
    # the vectors are certified to tol: residuals within its level on top of the rounding
    assert np.max(np.abs(A @ vt.T - u * s)) <= tol + 1e-13 * ref[0]
    assert np.max(np.abs(A.T @ u - vt.T * s)) <= tol + 1e-13 * ref[0]


def test_values_far_below_the_largest():
    """A spectrum down to 1e-15 sigma_1 takes the Sturm counts past the range of the minors' recurrence."""
    rng = np.random.default_rng(5)
    A = _matrix(40, 40, 10.0 ** -0.4, rng)
    u, s, vt, bnd = pg.svdp(A, 30, irl_mode=False, kmax=41, tol=1.0, delta=0.0, rng=np.random.default_rng(0))
    ref = np.linalg.svd(A, compute_uv=False)
    assert np.max(np.abs(s - ref[:30])) <= 64 * 40 * EPS * ref[0]


@pytest.mark.parametrize("scale", [1e-130, 1e-90, 1e90, 1e130])
def test_scaled_matrices(scale):
    """Matrices outside the scaled recurrence's range take the unscaled pivots; inside it, scaling changes nothing."""
    rng = np.random.default_rng(6)
    A = _matrix(30, 20, 0.8, rng)
    s1 = pg.svdp(A, 5, kmax=18, tol=1e-12, rng=np.random.default_rng(0))[1]
    s2 = pg.svdp(A * scale, 5, kmax=18, tol=1e-12, rng=np.random.default_rng(0))[1] / scale
    assert np.max(np.abs(s1 - s2)) <= 64 * 30 * EPS * s1[0]
