"""Gram-Schmidt over more columns than its kernels keep in shared memory at a
time (blocks of 64 columns in the projections, of 512 in the updates), for every
arithmetic and vector type, and the largest dimensions the drivers take.

k = 520 makes the first dimension 1041, on a matrix of rank 1100; delta = 0
projects every step on all columns before it.  Tolerances: a certified triplet
has a residual of at most tol sigma_1, the sums of up to m terms add at most
64 m eps sigma_1 (FP32 form, compensated sums: 64 sqrt(m) eps32)."""
import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg

pytestmark = pytest.mark.gpu

EPS, EPS32 = 2.0 ** -52, 2.0 ** -23
M, N, K = 1301, 1100, 520


def _matrix(m, n, per, seed, cplx, decay):
    rng = np.random.default_rng(seed)
    nnz = m * per
    val = rng.standard_normal(nnz) + (1j * rng.standard_normal(nnz) if cplx else 0.0)
    val = val * np.repeat((1.0 + np.arange(m)) ** -decay, per)
    return sp.csr_array((val, rng.integers(0, n, nnz).astype(np.int32), np.arange(m + 1) * per), shape=(m, n))


@pytest.mark.parametrize("form,arith", [("real", "planes"), ("real", "fp64"), ("real", "f3"), ("native", "planes"),
                                        ("native", "fp64"), ("block", "planes"), ("block", "fp64"), ("fp32", "planes")])
def test_blocks_of_columns(form, arith):
    cplx, f32 = form in ("native", "block"), form == "fp32"
    A = _matrix(M, N, 12, 5, cplx, 0.0 if f32 else 0.3)
    pg.set_cgs_arith(arith)
    pg.set_complex_form("block" if form == "block" else "native")
    try:
        u, s, vt, _ = pg.svdp(A, K, irl_mode=False, kmax=N, tol=1e-4 if f32 else 1e-12, delta=0.0,
                              precision="fp32" if f32 else "fp64", rng=np.random.default_rng(0))
    finally:
        pg.set_cgs_arith("planes")
        pg.set_complex_form("native")
    assert pg.get_stats()["nlandim"] > 1024
    lim = (1e-4 + 64 * np.sqrt(M) * EPS32 if f32 else 1e-12 + 64 * M * EPS) * s[0]
    v = vt.conj().T
    assert np.max(np.linalg.norm(A @ v - u * s, axis=0)) <= lim
    assert np.max(np.linalg.norm(A.conj().T @ u - v * s, axis=0)) <= lim
    assert np.max(np.abs(s - np.linalg.svd(A.toarray(), compute_uv=False)[:K])) <= lim


@pytest.mark.parametrize("form", ["real", "native", "block", "fp32"])
def test_largest_dimensions(form):
    m, kmax = 12001, 11500
    cplx, f32 = form in ("native", "block"), form == "fp32"
    A = _matrix(m, m, 5, 7, cplx, 0.9)
    pg.set_complex_form("block" if form == "block" else "native")
    try:
        u, s, vt, _ = pg.svdp(A, 2, irl_mode=False, kmax=kmax, tol=1e-4 if f32 else 1e-10, delta=0.0,
                              precision="fp32" if f32 else "fp64", rng=np.random.default_rng(0))
    finally:
        pg.set_complex_form("native")
        pg.release_memory()
    lim = (1e-4 + 64 * np.sqrt(m) * EPS32 if f32 else 1e-10 + 64 * m * EPS) * s[0]
    assert np.max(np.linalg.norm(A @ vt.conj().T - u * s, axis=0)) <= lim
