"""The chunked sparse product at the edges of its tiles: units past a multiple
of the unrolling, rows over many runs, empty rows and tiles, a last partial
tile, tiles shorter than a group; A x and A'y, real and complex, alone and
inside a solve.

Tolerance: a sum of k products in any order is off by at most
(k + 2) eps sum |a x| (complex: 4 (k + 2) eps).
"""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _rows(kind, m, rng):
    if kind.startswith("const"):
        return np.full(m, int(kind[5:]))
    if kind == "empty":
        return np.where(rng.random(m) < 0.7, 0, rng.integers(1, 9, m))
    if kind == "tiles":  # every third tile empty
        return np.where((np.arange(m) // 32) % 3 == 0, 0, rng.integers(1, 6, m))
    if kind == "long":   # a few rows over all runs of their tile
        cnt = rng.integers(0, 4, m)
        cnt[rng.integers(0, m, 1 + m // 40)] = rng.integers(50, 900, 1 + m // 40)
        return cnt
    return np.minimum(1 + (0.6 / rng.random(m)).astype(int), 1500)  # Zipf


def _matrix(kind, m, n, cplx, seed):
    rng = np.random.default_rng(seed)
    cnt = _rows(kind, m, rng)
    nnz = int(cnt.sum())
    val = rng.standard_normal(nnz) + (1j * rng.standard_normal(nnz) if cplx else 0.0)
    ptr = np.concatenate([[0], np.cumsum(cnt)])
    return sp.csr_array((val, rng.integers(0, n, nnz).astype(np.int32), ptr), shape=(m, n)), rng


def _vec(n, cplx, rng):
    return rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0.0)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m", [1, 31, 33, 4097])
@pytest.mark.parametrize("kind", ["const1", "const2", "const3", "const5", "const7", "const9", "empty", "tiles", "long",
                                  "zipf"])
def test_products(kind, m, cplx):
    n = 700
    A, rng = _matrix(kind, m, n, cplx, 7 * m + len(kind))
    op = pg.CsrOperator(A)
    # (abs(A) would add repeated entries first; the bound is on all of them)
    B = sp.csr_array((abs(A.data), A.indices.copy(), A.indptr.copy()), shape=A.shape)
    for y, x, M, P in ((op.matvec, _vec(n, cplx, rng), A, B), (op.rmatvec, _vec(m, cplx, rng), A.conj().T, B.T)):
        k = (np.diff(A.indptr) if P is B else np.bincount(A.indices, minlength=n)).max(initial=0)
        lim = (4 if cplx else 1) * (k + 2) * EPS * (P @ abs(x))
        # (the reference sum has the same bound)
        assert np.all(abs(np.asarray(y(x)) - M @ x) <= 2 * lim)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["const3", "empty", "long", "zipf"])
def test_solve(kind, cplx):
    A, _ = _matrix(kind, 3000, 2500, cplx, 5)
    u, s, vt, _ = pg.svdp(pg.CsrOperator(A), 4, kmax=40, tol=1e-12, delta=0.0, rng=np.random.default_rng(0))
    lim = (1e-12 + 64 * 3000 * 2 * EPS) * s[0]
    v = vt.conj().T
    assert np.max(np.linalg.norm(A @ v - u * s, axis=0)) <= lim
    assert np.max(np.linalg.norm(A.conj().T @ u - v * s, axis=0)) <= lim


@pytest.mark.parametrize("kmax", [30, 150])
def test_solve_with_a_full_grid(kmax):
    # enough rows to fill the chip: recurrences in shared (30) and in global memory (150)
    m = 80011
    A, _ = _matrix("zipf", m, m, False, 11)
    u, s, vt, _ = pg.svdp(pg.CsrOperator(A), 4, kmax=kmax, tol=1e-12, delta=0.0, rng=np.random.default_rng(0))
    lim = (1e-12 + 64 * m * 2 * EPS) * s[0]
    assert np.max(np.linalg.norm(A @ vt.T - u * s, axis=0)) <= lim
    assert np.max(np.linalg.norm(A.T @ u - vt.T * s, axis=0)) <= lim


def test_dimensions_of_two_threads():
    # a kernel's shared-memory limit belongs to the process: a small dimension
    # on one thread must not lower it under another thread's larger one
    A, _ = _matrix("zipf", 3000, 2500, False, 5)
    op = pg.CsrOperator(A)

    def values(kmax):
        return pg.svdp(op, 4, kmax=kmax, tol=1e-12, delta=0.0, rng=np.random.default_rng(0))[1]

    with ThreadPoolExecutor(1) as a, ThreadPoolExecutor(1) as b:
        first = a.submit(values, 290).result()
        for kmax in (12, 290, 30):
            small, again = b.submit(values, kmax), a.submit(values, 290)
            assert np.max(abs(small.result() - first)) <= (2e-12 + 128 * 3000 * EPS) * first[0]
            assert np.array_equal(again.result(), first)


@pytest.mark.parametrize("r", [1, 5, 33])
@pytest.mark.parametrize("m,n", [(40, 255), (300, 257), (40000, 5000)])
def test_low_rank_prepass(m, n, r):
    # rows of the thin factors shorter than a segment, at its edges, and cut over the grid
    S, rng = _matrix("const3", m, n, False, m + r)
    L, R, w = rng.standard_normal((m, r)), rng.standard_normal((n, r)), rng.standard_normal(r)
    op = pg.CsrOperator(S, sp.csr_array(L), sp.csr_array(R), w)
    B = sp.csr_array((abs(S.data), S.indices.copy(), S.indptr.copy()), shape=S.shape)
    for y, x, M, P, F, G in ((op.matvec, _vec(n, False, rng), S, B, L, R), (op.rmatvec, _vec(m, False, rng), S.T, B.T, R, L)):
        ref = M @ x + F @ (w * (G.T @ x))
        lim = (len(x) + r + 8) * EPS * (P @ abs(x) + abs(F) @ (abs(w) * (abs(G).T @ abs(x))))
        assert np.all(abs(np.asarray(y(x)) - ref) <= 2 * lim)
