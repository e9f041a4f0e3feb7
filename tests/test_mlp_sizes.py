"""The learned start's backward kernels at row counts around their tiles (32-row
stages and feature tiles, 64-row flushes, 128-row MMA tiles, chunks that end
early) against the CPU oracle, which rounds to BF16 at the same points.

Tolerance: the 2 % per block of the other gradient test (BF16 values whose FP32
sums land on the other side of a rounding boundary move by 2^-8)."""
import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg
from oracle import mlp_oracle as mo
from propack_gb300 import learned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k,pad", [(31, 2, 0), (33, 3, 1), (64, 4, 0), (65, 4, 0), (127, 5, 0),
                                     (129, 6, 2), (2431, 7, 0), (2433, 40, 0), (20011, 33, 3)])
def test_gradient_by_rows(m, k, pad):
    rng = np.random.default_rng(m)
    n = 50
    A = sp.csr_array((rng.standard_normal(4 * m), rng.integers(0, n, 4 * m).astype(np.int32), np.arange(m + 1) * 4),
                     shape=(m, n))
    op, model = pg.CsrOperator(A), learned.StartModel(seed=3)
    p = model.params.astype(np.float64)
    p[mo.OB1:mo.OW2] = 0.05
    p[mo.OB2:mo.OW3] = 0.05
    model.params = p
    buf = np.asfortranarray(rng.standard_normal((m + pad, k)) / np.sqrt(m))
    U = buf[:m]
    loss, g = model.grad(op, U)
    loss_o, g_o = mo.loss_and_grad(model.params, model.features(op), U, bf=True)
    assert abs(loss - loss_o) <= 1e-4 * abs(loss_o)
    for name, a, b in (("W1", mo.OW1, mo.OB1), ("b1", mo.OB1, mo.OW2), ("W2", mo.OW2, mo.OB2),
                       ("b2", mo.OB2, mo.OW3), ("w3", mo.OW3, mo.OB3), ("b3", mo.OB3, mo.NP)):
        err = np.linalg.norm(g[a:b] - g_o[a:b]) / max(np.linalg.norm(g_o[a:b]), 1e-30)
        assert err < 2e-2, (name, err)
    op.close()
    model.close()
