"""The learned start's sketch matrix (16 numbers per column of the operator) is
scratch of a call, not of the model: a wide operator's solve finds that memory
free."""
import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg
from propack_gb300 import learned

pytestmark = pytest.mark.gpu


def test_model_does_not_hold_the_sketch():
    torch = pytest.importorskip("torch")
    m, n = 1000, 8000000
    rng = np.random.default_rng(0)
    A = sp.csr_array((rng.standard_normal(5 * m), rng.integers(0, n, 5 * m).astype(np.int32), np.arange(m + 1) * 5),
                     shape=(m, n))
    model = learned.StartModel(seed=1)
    small = pg.CsrOperator(sp.csr_array(A[:, :1000]))
    model.features(small)
    op = pg.CsrOperator(A)
    pg.release_memory()
    free = torch.cuda.mem_get_info()[0]
    first = model.features(op)
    pg.release_memory()
    held = free - torch.cuda.mem_get_info()[0]
    assert held <= 8 * n + (1 << 28)
    # and the next calls, narrow and wide, find their own
    model.features(small)
    assert np.array_equal(model.features(op), first)
    op.close()
    small.close()
    model.close()
