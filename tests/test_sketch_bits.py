"""The learned start's sketch returns the same bits on every call: rows over the
whole-CTA threshold beside short ones, dozens of them in each CTA, and none.
Most entries of a row cancel in pairs of opposite sign, so that a sum taken in
another order differs far above the FP32 rounding of the features."""
import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg
from propack_gb300 import learned

pytestmark = pytest.mark.gpu


def _cancelling(rng, rows, per, n):
    """rows x per entries: pairs +a, -a in the same column and eight plain ones, in random order."""
    half = (per - 8) // 2
    a = rng.standard_normal((rows, half)) * 2.0 ** 30
    col = rng.integers(0, n, (rows, half))
    rest = per - 2 * half
    val = np.concatenate([a, -a, rng.standard_normal((rows, rest))], axis=1)
    idx = np.concatenate([col, col, rng.integers(0, n, (rows, rest))], axis=1)
    order = np.argsort(rng.random((rows, per)), axis=1)
    return np.take_along_axis(val, order, axis=1), np.take_along_axis(idx, order, axis=1)


@pytest.mark.parametrize("blocks,n", [
    ([(20, 40000)], 700),
    ([(257, 15000), (256, 15000)], 500),
    ([(9000, 12), (10, 1000), (700, 40)], 2000),
    ([(300, 100000)], 4000),
])
def test_same_bits(blocks, n):
    rng = np.random.default_rng(n)
    parts = [_cancelling(rng, rows, per, n) for per, rows in blocks]
    lens = np.concatenate([np.full(rows, per) for per, rows in blocks])
    ptr = np.concatenate([[0], np.cumsum(lens)])
    A = sp.csr_array((np.concatenate([v.ravel() for v, _ in parts]),
                      np.concatenate([i.ravel() for _, i in parts]).astype(np.int32), ptr), shape=(len(lens), n))
    op, model = pg.CsrOperator(A), learned.StartModel(seed=1)
    first = model.features(op)
    for _ in range(10):
        assert np.array_equal(model.features(op), first)
    op.close()
    model.close()
