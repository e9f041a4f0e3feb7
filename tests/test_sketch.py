"""The learned start's sketch and features on row lengths at the edges of its
kernel: empty and one-entry rows, rows around the whole-CTA threshold, more long
rows than one CTA's list holds, low-rank factors, and a second operator
that is wider than the first.

Tolerance: FP32 features of FP64 sums (the division by rho and the sums round in
FP64): two FP32 roundings relative to the row's norm."""
import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg
from propack_gb300 import learned
from test_learned_start import _omega

pytestmark = pytest.mark.gpu


def _csr(rng, lens, n):
    ptr = np.zeros(len(lens) + 1, dtype=np.int64)
    np.cumsum(lens, out=ptr[1:])
    return sp.csr_array((rng.standard_normal(int(ptr[-1])), rng.integers(0, n, int(ptr[-1])).astype(np.int32), ptr),
                        shape=(len(lens), n))


def _reference(A, lens, seed):
    Y = np.stack([A @ _omega(A.shape[1], c, seed) for c in range(16)], axis=1)
    nn = np.linalg.norm(Y, axis=1)
    rho = np.sqrt(np.mean(nn ** 2))
    rho = rho if rho > 0 else 1.0
    return np.concatenate([np.log1p(lens)[:, None] / 4.0, nn[:, None] / rho, 2 * Y / rho], axis=1)


@pytest.mark.parametrize("lens,n", [
    ([0, 1, 2, 3, 4, 5, 255, 256, 257, 0], 300),
    ([600] * 70 + [3] * 900, 400),
    ([300] * 3000, 500),
    (list(range(0, 40)) * 500, 100),
    ([7], 9),
])
def test_features_by_row_length(lens, n):
    rng = np.random.default_rng(len(lens))
    A = _csr(rng, lens, n)
    op, model = pg.CsrOperator(A), learned.StartModel(seed=1)
    ref = _reference(A, np.array(lens), model.sketch_seed)
    got = model.features(op)
    scale = np.maximum(np.abs(ref), ref[:, 1:2])
    assert np.max(np.abs(got - ref) / np.maximum(scale, 1e-30)) <= 2 * 2.0 ** -24
    op.close()
    model.close()


def test_low_rank_and_growing_operators():
    rng = np.random.default_rng(3)
    model = learned.StartModel(seed=1)
    for m, n, r in ((400, 300, 2), (3000, 2500, 5)):
        S = _csr(rng, rng.integers(0, 9, m), n)
        L, R = (sp.random_array((d, r), density=0.4, rng=rng, format="csr") for d in (m, n))
        w = 1.0 + np.arange(r)
        op = pg.CsrOperator(S, L, R, w)
        A = (S + (L * w) @ R.T).tocsr()
        lens = np.diff(S.indptr) + np.diff(sp.csr_array(L).indptr)
        ref = _reference(A, lens, model.sketch_seed)
        got = model.features(op)
        scale = np.maximum(np.abs(ref), ref[:, 1:2])
        assert np.max(np.abs(got - ref) / np.maximum(scale, 1e-30)) <= 2 * 2.0 ** -24
        op.close()
    model.close()
