"""A batch's device memory: the bases, one copy of the longest side of the
problems being solved at a time, the packed results.  A problem that is spread
over a cluster of CTAs takes no more of it than one that is not."""
import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg
from propack_gb300 import batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith", ["fp64", "planes"])
@pytest.mark.parametrize("m,n,nprob", [(1500000, 1500000, 1), (700000, 300001, 3)])
def test_footprint(m, n, nprob, arith):
    torch = pytest.importorskip("torch")
    dim, k = 24, 3
    rng = np.random.default_rng(m)
    mats = []
    for p in range(nprob):
        val = (rng.standard_normal(2 * m) * np.repeat((1.0 + np.arange(m)) ** -0.6, 2)).astype(np.float32)
        A = sp.csr_array((val.astype(np.float64), rng.integers(0, n, 2 * m).astype(np.int32), np.arange(m + 1) * 2),
                         shape=(m, n))
        A.sum_duplicates()
        mats.append(A)
    B = batch.Batch(mats)
    B.set_arith(arith)
    B.solve(k, kmax=dim, tol=1e-8, maxiter=2, u0=[np.ones(m)] * nprob, vectors=False)  # modules, tuning
    pg.release_memory()
    free = torch.cuda.mem_get_info()[0]
    sig, bnd, info, U, V = B.solve(k, kmax=dim, tol=1e-8, maxiter=60, u0=[np.ones(m)] * nprob)
    used = free - torch.cuda.mem_get_info()[0]
    B.close()
    pg.release_memory()
    basis = 8 * nprob * (m * (dim + 1) + n * dim) * (2 if arith == "planes" else 1)
    product = 8 * nprob * max(m, n) * (dim + 1)
    packed = 8 * nprob * max(m, n) * k
    # the pool grows in pieces; scratch that does not depend on the rows
    assert used <= basis + product + packed + (1 << 29)
    for p in range(nprob):
        if info[p] == 0:
            lim = (1e-8 + 64 * m * 2.0 ** -52) * sig[p][0]
            assert np.max(np.linalg.norm(mats[p] @ V[p] - U[p] * sig[p], axis=0)) <= lim
