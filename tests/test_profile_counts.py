"""propack_set_profiling counts each phase of a solve once, whether the products
come from the device operator (one launch per run of steps) or from the caller's
APROD (one launch per half step): no more products than the solve made, no more
time than the call took."""
import time

import numpy as np
import pytest
import scipy.sparse as sp
from scipy.sparse.linalg import aslinearoperator

import propack_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("host", [False, True])
def test_counted_once(host, cplx):
    rng = np.random.default_rng(3)
    A = sp.random_array((900, 500), density=0.02, rng=rng, format="csr")
    if cplx:
        A = sp.csr_array((A.data * np.exp(1j * A.data), A.indices, A.indptr), shape=A.shape)
    M = aslinearoperator(A) if host else pg.CsrOperator(A)
    kw = dict(irl_mode=False, kmax=300, tol=1e-6, delta=0.0)
    pg.svdp(M, 6, rng=np.random.default_rng(0), **kw)
    pg.set_profiling(True)
    try:
        t = time.perf_counter()
        pg.svdp(M, 6, rng=np.random.default_rng(0), **kw)
        t = time.perf_counter() - t
        nopx, prof = pg.get_stats()["nopx"], pg.get_profile()
    finally:
        pg.set_profiling(False)
    products = prof["spmv_adj"][0] + prof["spmv_fwd"][0]
    assert 20 <= products <= nopx
    assert sum(ms for _, ms in prof.values()) <= 1e3 * t
