"""Batches whose problems are spread over clusters of CTAs: one large problem
alone, a few uneven ones (the smallest shorter than the cluster's threads),
restarts, both arithmetics, results with and without vectors, problems that do
not converge beside others that do.

Tolerances: values converged to tol = 1e-12 with full reorthogonalisation, so
within tol plus 64 m eps of the dense SVD; residuals the same."""
import numpy as np
import pytest
import scipy.sparse as sp

from propack_gb300 import batch

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _matrix(rng, m, n, per_row):
    val = rng.standard_normal(m * per_row) * np.repeat((1.0 + np.arange(m)) ** -0.6, per_row)
    A = sp.csr_array((val.astype(np.float32).astype(np.float64), rng.integers(0, n, m * per_row).astype(np.int32),
                      np.arange(m + 1) * per_row), shape=(m, n))
    A.sum_duplicates()
    A.data = A.data.astype(np.float32).astype(np.float64)
    return A


def _check(A, s, U, V, tol):
    lim = (tol + 64 * max(A.shape) * EPS) * s[0]
    assert np.max(np.linalg.norm(A @ V - U * s, axis=0)) <= lim
    assert np.max(np.linalg.norm(A.T @ U - V * s, axis=0)) <= lim
    G = (A.T @ A).toarray() if A.shape[1] <= A.shape[0] else (A @ A.T).toarray()
    ref = np.sqrt(np.maximum(np.linalg.eigvalsh(G)[::-1][:len(s)], 0))
    # the Gram matrix squares the condition: eps sigma_1^2 / sigma_i on each value
    assert np.all(np.abs(s - ref) <= lim + 64 * max(A.shape) * EPS * ref[0] ** 2 / ref)


@pytest.mark.parametrize("arith", ["fp64", "planes"])
@pytest.mark.parametrize("shapes", [
    [(12000, 3000, 40)],                                    # eight CTAs
    [(9000, 1201, 30), (6001, 2000, 30), (70, 50, 5)],      # uneven, the last shorter than a cluster
    [(1500, 3001, 200), (3000, 1501, 100), (40, 33, 4)],    # wide and tall
    [(2000, 600, 41)] * 3,
])
def test_clusters(shapes, arith):
    rng = np.random.default_rng(len(shapes))
    mats = [_matrix(rng, *s) for s in shapes]
    u0 = [rng.uniform(size=A.shape[0]) for A in mats]
    B = batch.Batch(mats)
    B.set_arith(arith)
    sig, bnd, info, U, V = B.solve(5, kmax=24, tol=1e-12, maxiter=100, u0=u0)
    assert np.all(info == 0)
    if arith == "fp64":
        assert B.stats["fallback"] == 0 and B.stats["grid"] > len(mats)
    for p, A in enumerate(mats):
        _check(A, sig[p], U[p], V[p], 1e-12)
    sig2 = B.solve(5, kmax=24, tol=1e-12, maxiter=100, u0=u0, vectors=False)[0]
    assert np.array_equal(sig, sig2)
    B.close()


def test_unconverged_problems_beside_converged_ones():
    """maxiter = 1: the flat spectrum does not converge, its part of U and V stays zero."""
    rng = np.random.default_rng(9)
    flat = sp.csr_array((np.ones(60000, dtype=np.float32) * rng.choice([-1.0, 1.0], 60000),
                         rng.integers(0, 2000, 60000).astype(np.int32), np.arange(6001) * 10), shape=(6000, 2000))
    mats = [_matrix(rng, 5000, 1000, 20), flat, _matrix(rng, 4000, 900, 20)]
    u0 = [rng.uniform(size=A.shape[0]) for A in mats]
    B = batch.Batch(mats)
    sig, bnd, info, U, V = B.solve(3, kmax=40, tol=1e-10, maxiter=1, u0=u0)
    assert info.tolist() == [0, -1, 0]
    for p in (0, 2):
        _check(mats[p], sig[p], U[p], V[p], 1e-10)
    assert not U[1].any() and not V[1].any()
    B.close()
