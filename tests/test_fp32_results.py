"""The single-precision drivers hand their FP32 vectors out as they are: the
same solve through the FP64-typed entry point (precision "fp32") returns the
same numbers widened, bit for bit, whatever the leading dimensions."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("irl", [True, False])
@pytest.mark.parametrize("m,n,pad", [(33, 20, 0), (1001, 517, 3), (4099, 4096, 1), (300007, 20001, 5)])
def test_same_bits_as_the_widened_results(m, n, pad, irl):
    rng = np.random.default_rng(m)
    val = rng.standard_normal(5 * m) * np.repeat((1.0 + np.arange(m)) ** -0.7, 5)
    A = sp.csr_array((val, rng.integers(0, n, 5 * m).astype(np.int32), np.arange(m + 1) * 5), shape=(m, n))
    k, kmax = 4, 18
    v0 = rng.uniform(size=m).astype(np.float32)
    op = pg.CsrOperator(A)
    u, s, vt, bnd = pg.svdp(op, k, irl_mode=irl, kmax=kmax, tol=1e-5, v0=v0.astype(np.float64), precision="fp32",
                            rng=np.random.default_rng(0))
    L, ci = pg.load(), lambda v: C.byref(C.c_int(v))
    p = lambda a: C.c_void_p(a.ctypes.data)
    U = np.full((m + pad, kmax + 1), 7.0, dtype=np.float32, order="F")
    V = np.full((n + pad, kmax), 7.0, dtype=np.float32, order="F")
    U[:m, 0] = v0
    sig, bb = np.zeros(k, dtype=np.float32), np.zeros(k, dtype=np.float32)
    lwork, liwork, _ = pg.work_sizes(m, n, kmax, irl=irl)
    work, iwork = np.empty(lwork, dtype=np.float32), np.empty(liwork, dtype=np.int32)
    # svdp's defaults, the drivers raise them to the FP32 levels
    eps = np.finfo(np.float64).eps
    dop, iop = np.array([eps ** 0.5, eps ** 0.75, 0.0, 0.002], dtype=np.float32), np.array([0, 1], dtype=np.int32)
    ne, info, par = C.c_int(k), C.c_int(0), np.zeros(1, dtype=np.float32)
    tail = (p(work), ci(lwork), p(iwork), ci(liwork), p(dop), p(iop), C.byref(info), p(par), p(op.iparm))
    tol = C.byref(C.c_float(1e-5))
    if irl:
        L.slansvd_irl_(b"L", b"y", b"y", ci(m), ci(n), ci(kmax), ci(kmax - k), C.byref(ne), ci(1000),
                       L.propack_gpu_csr_saprod_, p(U), ci(m + pad), p(sig), p(bb), p(V), ci(n + pad), tol, *tail,
                       C.c_size_t(1), C.c_size_t(1), C.c_size_t(1))
    else:
        L.slansvd_(b"y", b"y", ci(m), ci(n), C.byref(ne), ci(kmax), L.propack_gpu_csr_saprod_, p(U), ci(m + pad),
                   p(sig), p(bb), p(V), ci(n + pad), tol, *tail, C.c_size_t(1), C.c_size_t(1))
    op.close()
    assert info.value == 0 and ne.value == k
    assert np.array_equal(U[:m, :k].astype(np.float64), u)
    assert np.array_equal(V[:n, :k].T.astype(np.float64), vt)
    assert np.all(U[m:] == 7.0) and np.all(V[n:] == 7.0) and np.all(V[:, k:] == 7.0)
