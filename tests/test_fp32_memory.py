"""The FP32 form's results through the FP64-typed entry point are widened in the
memory that the solve already holds, and in as many pieces as that takes: few
and many wanted columns of a long and of a short side, bit for bit the
single-precision driver's values."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg

pytestmark = pytest.mark.gpu


def _matrix(m, n, per, seed):
    rng = np.random.default_rng(seed)
    val = rng.standard_normal(per * m) * np.repeat((1.0 + np.arange(m)) ** -0.7, per)
    return sp.csr_array((val, rng.integers(0, n, per * m).astype(np.int32), np.arange(m + 1) * per), shape=(m, n))


def test_footprint():
    torch = pytest.importorskip("torch")
    m, n, k, kmax = 3000000, 2000000, 20, 80
    op = pg.CsrOperator(_matrix(m, n, 2, 1))
    kw = dict(irl_mode=False, kmax=kmax, tol=1e-3, precision="fp32")
    pg.svdp(op, 1, rng=np.random.default_rng(0), **kw)
    pg.release_memory()
    free = torch.cuda.mem_get_info()[0]
    pg.svdp(op, k, rng=np.random.default_rng(0), **kw)
    used = free - torch.cuda.mem_get_info()[0]
    op.close()
    pg.release_memory()
    bases = 4 * (m + n) * (kmax + 1)
    product = 4 * max(m, n) * (kmax + 1)
    vectors = 24 * max(m, n)
    assert used <= bases + product + vectors + (1 << 29)


@pytest.mark.parametrize("m,n,k,kmax", [(900, 45, 40, 45), (70, 900, 60, 70), (500, 34, 33, 34), (5001, 64, 8, 64)])
def test_pieces(m, n, k, kmax):
    A = _matrix(m, n, 6, m)
    v0 = np.random.default_rng(1).uniform(size=m).astype(np.float32)
    op = pg.CsrOperator(A)
    L, ci = pg.load(), lambda v: C.byref(C.c_int(v))
    p = lambda a: C.c_void_p(a.ctypes.data)
    eps = np.finfo(np.float64).eps

    def run(single):
        ty = np.float32 if single else np.float64
        U, V = np.zeros((m, kmax + 1), dtype=ty, order="F"), np.zeros((n, kmax), dtype=ty, order="F")
        U[:, 0] = v0
        sig, bnd = np.zeros(k, dtype=ty), np.zeros(k, dtype=ty)
        lwork, liwork, _ = pg.work_sizes(m, n, kmax, irl=False)
        work, iwork = np.empty(lwork, dtype=ty), np.empty(liwork, dtype=np.int32)
        dop, iop = np.array([eps ** 0.5, eps ** 0.75, 0.0], dtype=ty), np.array([0, 1], dtype=np.int32)
        ne, info, par = C.c_int(k), C.c_int(0), np.zeros(1, dtype=ty)
        tol = C.byref((C.c_float if single else C.c_double)(1e-3))
        f, ap = (L.slansvd_, L.propack_gpu_csr_saprod_) if single else (L.dlansvd_, L.propack_gpu_csr_aprod_)
        f(b"y", b"y", ci(m), ci(n), C.byref(ne), ci(kmax), C.cast(ap, C.c_void_p), p(U), ci(m), p(sig), p(bnd), p(V),
          ci(n), tol, p(work), ci(lwork), p(iwork), ci(liwork), p(dop), p(iop), C.byref(info), p(par), p(op.iparm),
          C.c_size_t(1), C.c_size_t(1))
        return U, V, ne.value, info.value

    us, vs, ks, infos = run(True)
    pg.set_precision("fp32")
    try:
        ud, vd, kd, infod = run(False)
    finally:
        pg.set_precision("fp64")
        op.close()
    # (a Krylov space as large as the matrix: all k converge, in one to two pieces per side)
    assert (ks, infos) == (kd, infod) == (k, 0)
    assert np.array_equal(us[:, :k].astype(np.float64), ud[:, :k])
    assert np.array_equal(vs[:, :k].astype(np.float64), vd[:, :k])
