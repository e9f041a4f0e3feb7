"""The restart and Ritz products of the implicitly restarted driver: the
longer basis changes places with the product's buffer, the shorter one is
copied back; with a million rows the product leaves for the host in row chunks
while the other side's is formed.

Tolerances: a certified triplet has a residual of at most tol sigma_1, and the
sums of up to m terms in its products add at most 64 m eps sigma_1; the basis
is kept orthogonal to eps (delta = 0), so the vectors are orthonormal to the
same level over sigma_1.
"""
import threading

import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _matrix(m, n, nnz, seed, cplx):
    rng = np.random.default_rng(seed)
    val = rng.standard_normal(nnz) + (1j * rng.standard_normal(nnz) if cplx else 0.0)
    row = rng.integers(0, m, nnz)
    return sp.csr_array(sp.coo_array((val * (1.0 + row) ** -0.3, (row, rng.integers(0, n, nnz))), shape=(m, n)))


def _check(m, n, cplx):
    A = _matrix(m, n, 6 * max(m, n), m + 3 * n, cplx)
    k, tol = 4, 1e-11
    u, s, vt, _ = pg.svdp(A, k, irl_mode=True, kmax=16, tol=tol, delta=0.0, rng=np.random.default_rng(0))
    lim = tol + 64 * max(m, n) * EPS
    v = vt.conj().T
    assert np.max(np.linalg.norm(A @ v - u * s, axis=0)) <= lim * s[0]
    assert np.max(np.linalg.norm(A.conj().T @ u - v * s, axis=0)) <= lim * s[0]
    assert np.max(np.abs(u.conj().T @ u - np.eye(k))) <= lim
    assert np.max(np.abs(v.conj().T @ v - np.eye(k))) <= lim


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n", [(400, 400), (401, 415), (416, 417), (5000, 900), (900, 5000), (4130, 4100)])
def test_longer_and_shorter_side(m, n, cplx):
    _check(m, n, cplx)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n", [((1 << 20) + 5, (1 << 20) + 5), ((1 << 20) + 33, 700), (700, (1 << 20) + 33)])
def test_chunks_to_the_host(m, n, cplx):
    _check(m, n, cplx)


def test_threads_and_release():
    # streams, events and pinned words of one call serve the next; concurrent
    # calls have one set each, and a release between calls only frees idle ones
    errs = []

    def work(i):
        try:
            for _ in range(3):
                _check(600 + 50 * i, 500, False)
                pg.release_memory()
        except BaseException as e:  # noqa: BLE001
            errs.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(10)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errs
