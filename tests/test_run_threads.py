"""Cooperative launches of the run kernel from two threads whose dimensions want
different carve-outs of the same kernel: with a grid that fills the chip, the
larger dimension's launches must find their own carve-out again whatever the
other thread asked for in between.  The grid follows from the size and the
dimension alone, so every solve repeats the serial one bit for bit."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest
import scipy.sparse as sp

import propack_gb300 as pg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule,m,large", [("chunked", 70000, 150), ("chunked", 70000, 290), ("staged", 80000, 300),
                                              ("chunked", 90000, 1100)])
def test_carve_outs_of_two_threads(schedule, m, large):
    rng = np.random.default_rng(m)
    val = rng.standard_normal(5 * m) * np.repeat((1.0 + np.arange(m)) ** -0.4, 5)
    A = sp.csr_array((val, rng.integers(0, m, 5 * m).astype(np.int32), np.arange(m + 1) * 5), shape=(m, m))
    pg.set_spmv_schedule(schedule)
    try:
        op = pg.CsrOperator(A)
    finally:
        pg.set_spmv_schedule("rule")

    def solve(kmax, k):
        u, s, vt, _ = pg.svdp(op, k, irl_mode=False, kmax=kmax, tol=1e-9, rng=np.random.default_rng(0))
        return u, s, vt

    def same(a, b):
        return all(np.array_equal(x, y) for x, y in zip(a, b))

    with ThreadPoolExecutor(1) as one, ThreadPoolExecutor(1) as two:
        big, small = one.submit(solve, large, 4).result(), {q: two.submit(solve, q, 1).result() for q in (30, 40)}
        for q in small:
            # in turn: `one` launches under what it last asked for unless it asks again
            assert same(two.submit(solve, q, 1).result(), small[q])
            assert same(one.submit(solve, large, 4).result(), big)
        for _ in range(3):  # at once
            jobs = [(two.submit(solve, 30, 1), small[30]), (one.submit(solve, large, 4), big)]
            assert all(same(j.result(), want) for j, want in jobs)
    op.close()
