"""The Lanczos run kernel at the edges of its grid and of its phases: one CTA
and many, chunks of the projections that are split by rows, by columns or by
both, partial sums reduced by one CTA or by the grid, recurrences in shared
and in global memory, every Gram-Schmidt arithmetic, products of the device
operator (both schedules) and of a host callback.

Tolerances: a certified triplet has a residual of at most tol sigma_1; the
sums of up to m terms in its products and inner products add at most
64 m eps sigma_1 (FP32 form, whose sums are compensated: 64 sqrt(m) eps32).
With partial reorthogonalisation (delta > 0) the basis is orthogonal to
sqrt(eps) only and the vectors' residuals are not held to that level (the
reference's own are 1e-11 on these inputs); the values are.
"""
import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import aslinearoperator

import propack_gb300 as pg

pytestmark = pytest.mark.gpu

EPS, EPS32 = 2.0 ** -52, 2.0 ** -23


def _matrix(m, n, nnz_row, seed, cplx=False):
    rng = np.random.default_rng(seed)
    nnz = m * nnz_row
    val = rng.standard_normal(nnz) + (1j * rng.standard_normal(nnz) if cplx else 0.0)
    val = val * np.repeat((1.0 + np.arange(m)) ** -0.7, nnz_row)
    return sp.csr_array((val, rng.integers(0, n, nnz).astype(np.int32), np.arange(m + 1) * nnz_row), shape=(m, n))


def _check(A, k, tol, level, **kw):
    u, s, vt, bnd = pg.svdp(A, k, tol=tol, rng=np.random.default_rng(0), **kw)
    B = A if sp.issparse(A) else A.A
    lim = (tol + level) * s[0]
    if kw.get("delta") == 0.0 or kw.get("precision") == "fp32":
        assert np.max(np.linalg.norm(B @ vt.conj().T - u * s, axis=0)) <= lim
        assert np.max(np.linalg.norm(B.conj().T @ u - vt.conj().T * s, axis=0)) <= lim
    if max(B.shape) <= 3000:
        ref = np.linalg.svd(B.toarray(), compute_uv=False)[:k]
        assert np.max(np.abs(s - ref)) <= lim
    return s


@pytest.mark.parametrize("arith", ["planes", "fp64", "f3"])
@pytest.mark.parametrize("m,n", [(127, 40), (128, 128), (129, 300), (2049, 511), (513, 2100)])
def test_sizes_and_arithmetics(m, n, arith):
    A = _matrix(m, n, 4, m + n)
    pg.set_cgs_arith(arith)
    try:
        for delta in (None, 0.0):
            k = min(4, n // 4)
            _check(A, k, 1e-12, 64 * max(m, n) * EPS, kmax=min(40, min(m, n)), delta=delta)
    finally:
        pg.set_cgs_arith("planes")


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n", [(8191, 6000), (16384, 16385), (33001, 9001), (70001, 90001)])
def test_chunks_and_reductions(m, n, cplx):
    """delta = 0: every step projects on all columns, up to 48 of them over 64 to 608 CTAs."""
    _check(_matrix(m, n, 5, m, cplx), 6, 1e-12, 64 * max(m, n) * EPS, kmax=48, delta=0.0)


@pytest.mark.parametrize("kmax", [299, 300, 301, 420])
def test_recurrences_beyond_shared_memory(kmax):
    _check(_matrix(1500, 1100, 6, kmax), 60, 1e-12, 64 * 1500 * EPS, kmax=kmax)


@pytest.mark.parametrize("m,n", [(129, 60), (3000, 2001), (40003, 20001)])
def test_fp32_form(m, n):
    _check(_matrix(m, n, 5, n), 4, 1e-6, 64 * np.sqrt(max(m, n)) * EPS32, kmax=32, precision="fp32")


@pytest.mark.parametrize("schedule", ["chunked", "staged"])
def test_schedules(schedule):
    A = _matrix(5003, 3001, 40, 3)
    pg.set_spmv_schedule(schedule)
    try:
        op = pg.CsrOperator(A)
        u, s, vt, bnd = pg.svdp(op, 6, kmax=36, tol=1e-12, delta=0.0, rng=np.random.default_rng(0))
        op.close()
    finally:
        pg.set_spmv_schedule("rule")
    assert np.max(np.linalg.norm(A @ vt.T - u * s, axis=0)) <= (1e-12 + 64 * 5003 * EPS) * s[0]


@pytest.mark.parametrize("cplx", [False, True])
def test_host_products(cplx):
    A = _matrix(700, 400, 5, 11, cplx)
    kw = dict(kmax=30, tol=1e-12)
    s0 = pg.svdp(A, 5, rng=np.random.default_rng(0), **kw)[1]
    s1 = pg.svdp(aslinearoperator(A), 5, rng=np.random.default_rng(0), **kw)[1]
    assert np.max(np.abs(s0 - s1)) <= 64 * 700 * EPS * s0[0]


def test_low_rank_prepass():
    """Factors with empty, one-entry and long columns (segments of the prepass)."""
    rng = np.random.default_rng(2)
    m, n, r = 5000, 1300, 5
    S = _matrix(m, n, 4, 7)
    L = sp.random_array((m, r), density=0.2, rng=rng, format="csr").tolil()
    R = sp.random_array((n, r), density=0.3, rng=rng, format="csr").tolil()
    L[:, 0] = rng.standard_normal((m, 1))
    R[:, 0] = rng.standard_normal((n, 1))
    L[:, 1] = 0.0
    R[:, 2] = 0.0
    R[7, 2] = 1.0
    L, R = sp.csr_array(L), sp.csr_array(R)
    w = np.array([3.0, 1.0, 2.0, 0.5, 0.25]) / 50.0
    op = pg.CsrOperator(S, L, R, w)
    A = (S + (L * w) @ R.T).tocsr()
    x, y = rng.standard_normal(n), rng.standard_normal(m)
    np.testing.assert_allclose(op.matvec(x), A @ x, rtol=0, atol=64 * m * EPS * np.abs(A @ x).max())
    np.testing.assert_allclose(op.rmatvec(y), A.T @ y, rtol=0, atol=64 * m * EPS * np.abs(A.T @ y).max())
    u, s, vt, bnd = pg.svdp(op, 5, kmax=30, tol=1e-12, delta=0.0, rng=np.random.default_rng(0))
    op.close()
    assert np.max(np.linalg.norm(A @ vt.T - u * s, axis=0)) <= (1e-12 + 64 * m * EPS) * s[0]
    assert np.max(np.linalg.norm(A.T @ u - vt.T * s, axis=0)) <= (1e-12 + 64 * m * EPS) * s[0]
