"""The work that users of this framework have it do, as cases with seeded inputs.

Every case is one call through the package's public entry points: a truncated
SVD by the plain or the restarted driver (FP64, mixed, single precision,
complex*16, from a kept device operator or straight from a scipy matrix),
thousands of small problems in one batched solve, the learned start vector's
inference and training gradient, and the products of the device operator.
Sizes and spectra are those of the benchmark's workloads and of the tests,
scaled; the wanted triplets are separated from the rest of the spectrum, as
they are where singular vectors are asked for, and the tolerances are tight
enough that the vectors are determined by the input to many digits.
"""
import ctypes as C
import math
import mmap

import numpy as np
import scipy.sparse as sp
import torch

import propack_gb300 as pg
from propack_gb300 import batch as pg_batch
from propack_gb300 import learned as pg_learned


def listed():
    return [
        # the reference's CPU-sized problem: dlansvd on a 2000 x 1000 matrix, latency all the way
        dict(name="lansvd 2000x1000", kind="lansvd", m=2000, n=1000, nnz_row=5, k=10, kmax=200),
        # the drop-in call of a scipy user: svdp(A, k) on a host matrix, default tolerance, restarts
        dict(name="svdp scipy 20011x4999", kind="svdp", m=20011, n=4999, nnz_row=10, k=10, kmax=40),
        # a mid-size factored operator (the matrix family of the learned start), restarted
        dict(name="irl factored 200000x50000", kind="factored", m=200_000, n=50_000, nnz_row=10, rank=32, udens=1.0,
             vdens=1.0, w0=50.0, decay=0.9, noise=0.1, k=16, kmax=32),
        # a large factored operator with sparse factors, k = 50 and Lanczos dimension 150
        dict(name="irl factored 1000003x250007", kind="factored", m=1_000_003, n=250_007, nnz_row=20, rank=64,
             udens=0.01, vdens=0.05, w0=100.0, decay=0.97, noise=1.0, k=50, kmax=150),
        # the headline: a 4M x 4M matrix with Zipf row lengths in FP64
        dict(name="irl zipf 4000000", kind="zipf", m=4_000_000, k=50, kmax=150, precision="fp64"),
        # the same family in the mixed form (FP32 vectors, FP64 refinement)
        dict(name="mixed zipf 1000000", kind="zipf", m=1_000_000, k=20, kmax=60, precision="mixed"),
        # the REAL driver slansvd_irl_ of a single-precision program
        dict(name="single zipf 500001", kind="single", m=500_001, k=10, kmax=40),
        # the complex*16 driver
        dict(name="complex zipf 1000000", kind="complex", m=1_000_000, k=20, kmax=60),
        # many small problems of uneven size in one call
        dict(name="batch 192", kind="batch", nprob=192, k=8, kmax=40),
        # the learned start vector: training gradient (forward and backward) and the proposal (forward alone)
        dict(name="learned grad 200000", kind="learned", m=200_000, n=50_000, nnz_row=10, k=32, grad=True),
        dict(name="learned start 50000", kind="learned", m=50_000, n=12_500, nnz_row=10, k=32, grad=False),
        # A x and A'y on device vectors, without allocation
        dict(name="apply 1000000", kind="apply", m=1_000_000, n=500_009, mean=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: every kind as often, sizes spread over the range that the listed ones stand for."""
    kind = rng.choice(["lansvd", "svdp", "factored", "zipf", "zipf", "single", "complex", "batch", "learned", "apply"])
    if kind == "lansvd":
        m = _log(rng, 1500, 8000)
        return dict(kind=kind, m=m, n=max(800, m // rng.choice([1, 2, 3])), nnz_row=rng.randint(4, 12),
                    k=rng.randint(4, 10), kmax=200)
    if kind == "svdp":
        m = _log(rng, 5000, 100_000)
        k = rng.randint(4, 12)
        return dict(kind=kind, m=m, n=max(2000, m // rng.choice([1, 2, 4])), nnz_row=rng.randint(5, 20), k=k,
                    kmax=4 * k)
    if kind == "factored":
        m = _log(rng, 30_000, 700_000)
        k = rng.randint(8, 20)
        return dict(kind=kind, m=m, n=m // rng.randint(2, 5), nnz_row=rng.randint(5, 20), rank=32, udens=0.05,
                    vdens=0.1, w0=100.0, decay=0.9, noise=0.1, k=k, kmax=rng.choice([2, 3]) * k)
    if kind == "zipf":
        k = rng.randint(8, 50)
        precision = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, m=_log(rng, 50_000, 2_000_000 if precision == "fp64" else 800_000),
                    k=k, kmax=3 * k, precision=precision)
    if kind == "single":
        k = rng.randint(5, 15)
        return dict(kind=kind, m=_log(rng, 20_000, 1_000_000), k=k, kmax=4 * k)
    if kind == "complex":
        k = rng.randint(5, 30)
        return dict(kind=kind, m=_log(rng, 20_000, 1_500_000), k=k, kmax=3 * k)
    if kind == "batch":
        return dict(kind=kind, nprob=_log(rng, 16, 256), k=rng.randint(4, 10), kmax=40)
    if kind == "learned":
        m = _log(rng, 5000, 400_000)
        return dict(kind=kind, m=m, n=max(1000, m // 4), nnz_row=rng.randint(5, 15), k=rng.randint(8, 32),
                    grad=rng.choice([True, False]))
    m = _log(rng, 2000, 4_000_000)
    return dict(kind="apply", m=m, n=max(1000, int(m * rng.uniform(0.2, 1.2))), mean=rng.choice([5, 8, 20, 60]))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _uniform_rows(g, m, n, nnz_row, scale):
    """m x n CSR with nnz_row uniform columns per row (as drawn) and N(0, scale^2) values."""
    idx = torch.randint(0, n, (m * nnz_row,), generator=g, device="cuda", dtype=torch.int32)
    val = torch.randn(m * nnz_row, generator=g, device="cuda", dtype=torch.float64) * scale
    ptr = np.arange(m + 1, dtype=np.int64) * nnz_row
    return sp.csr_array((val.cpu().numpy(), idx.cpu().numpy(), ptr), shape=(m, n))


def _unit_columns(g, rows, r, dens):
    """rows x r CSR, each column `dens` dense with Gaussian entries and of unit norm."""
    D = torch.randn(rows, r, generator=g, device="cuda", dtype=torch.float64)
    if dens < 1.0:
        D *= torch.rand(rows, r, generator=g, device="cuda") < dens
    D /= D.norm(dim=0)
    row, col = torch.nonzero(D, as_tuple=True)
    ptr = np.zeros(rows + 1, dtype=np.int64)
    np.cumsum(torch.bincount(row, minlength=rows).cpu().numpy(), out=ptr[1:])
    return sp.csr_array((D[row, col].cpu().numpy(), col.to(torch.int32).cpu().numpy(), ptr), shape=(rows, r))


def _decaying(g, m, n, nnz_row):
    """Uniform rows, row i scaled by (1 + i)^-1/2: the reference workload's decaying spectrum."""
    A = _uniform_rows(g, m, n, nnz_row, 1.0)
    A.data *= np.repeat((1.0 + np.arange(m)) ** -0.5, nnz_row)
    return A


def _zipf(g, m, cplx=False, lo=4, hi=2000):
    """m x m CSR, Zipf(2) row lengths in [lo, hi], uniform columns, N(0, 1) (1 + i mod 1000)^-0.7 values that
    FP32 holds exactly (complex: real and imaginary parts)."""
    u = torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
    cnt = torch.clamp(torch.floor(0.6079 / torch.clamp(u, min=1e-7)), lo, hi).to(torch.int64)
    nnz = int(cnt.sum())
    ptr = np.zeros(m + 1, dtype=np.int64)
    np.cumsum(cnt.cpu().numpy(), out=ptr[1:])
    idx = torch.randint(0, m, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    w = torch.repeat_interleave((1.0 + torch.arange(m, device="cuda") % 1000) ** -0.7, cnt)
    val = torch.randn((2, nnz) if cplx else nnz, generator=g, device="cuda") * w
    val = torch.complex(val[0].double(), val[1].double()) if cplx else val.double()
    return sp.csr_array((val.cpu().numpy(), idx.cpu().numpy(), ptr), shape=(m, m))


def _matrix(case, seed):
    """The host matrix of a solver case: (S, L, R, w), L, R, w None where the operator is S alone."""
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("lansvd", "svdp"):
        return _decaying(g, case["m"], case["n"], case["nnz_row"]), None, None, None
    if kind == "factored":
        m, n, r = case["m"], case["n"], case["rank"]
        S = _uniform_rows(g, m, n, case["nnz_row"], case["noise"])
        L, R = _unit_columns(g, m, r, case["udens"]), _unit_columns(g, n, r, case["vdens"])
        return S, L, R, case["w0"] * case["decay"] ** np.arange(r)
    return _zipf(g, case["m"], cplx=kind == "complex"), None, None, None


def _start(seed, m, cplx=False):
    g = _gen(seed + 1_000_003)
    u = torch.rand(m, generator=g, device="cuda", dtype=torch.complex128 if cplx else torch.float64)
    return u.cpu().numpy()


def _batch_mats(case, seed):
    """Uneven sparse matrices, m in [500, 20000], n in [200, 8000], 1 % dense, values that FP32 holds, rows scaled so
    that the leading values are separated.  The sizes are the case's, the entries the seed's."""
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(case["nprob"])
    mats = []
    for _ in range(case["nprob"]):
        m, n = int(sizes.integers(500, 20_001)), int(sizes.integers(200, 8001))
        cnt = np.maximum(1, rng.binomial(n, 0.01, size=m)).astype(np.int64)
        ptr = np.zeros(m + 1, dtype=np.int64)
        np.cumsum(cnt, out=ptr[1:])
        nnz = int(ptr[-1])
        val = rng.standard_normal(nnz, dtype=np.float32)
        val *= np.repeat((1.0 + np.arange(m)) ** -0.5, cnt).astype(np.float32)
        A = sp.csr_array((val.astype(np.float64), rng.integers(0, n, size=nnz, dtype=np.int32), ptr), shape=(m, n))
        mats.append(A)
    return mats


def _tol(case):
    return {"lansvd": 1e-12, "svdp": 0.0, "single": 1e-6, "batch": 1e-11}.get(case["kind"], 1e-12)


def _array(rows, cols, typ):
    """A zeroed column-major array on pages of its own."""
    buf = mmap.mmap(-1, rows * cols * np.dtype(typ).itemsize)
    return np.frombuffer(buf, dtype=typ).reshape((rows, cols), order="F")


class _Locked:
    """Page-locks an array's memory for as long as it lives."""

    def __init__(self, a):
        self.array, self.rt = a, torch.cuda.cudart()
        torch.cuda.init()
        rc = int(self.rt.cudaHostRegister(a.ctypes.data, a.shape[0] * a.shape[1] * a.itemsize, 0))
        if rc != 0:
            raise RuntimeError(f"cudaHostRegister failed ({rc})")

    def __del__(self):
        torch.cuda.synchronize()
        self.rt.cudaHostUnregister(self.array.ctypes.data)


class _State:
    """A case's inputs and handles; the device operator goes with it."""

    def __init__(self, case, seed):
        self.case, self.seed = case, seed


def prepare(case, seed):
    st = _State(case, seed)
    kind = case["kind"]
    if kind == "batch":
        mats = _batch_mats(case, seed)
        st.batch = pg_batch.Batch(mats)
        k, np_ = case["k"], len(mats)
        st.u0 = np.random.default_rng(seed + 1).uniform(size=int(st.batch.m.sum()))
        st.sigma, st.bnd, st.info = np.zeros((np_, k)), np.zeros((np_, k)), np.zeros(np_, dtype=np.int32)
        st.U, st.V = np.zeros(int(st.batch.m.sum()) * k), np.zeros(int(st.batch.n.sum()) * k)
        return st
    if kind == "learned":
        g = _gen(seed)
        m, n, k = case["m"], case["n"], case["k"]
        S = _uniform_rows(g, m, n, case["nnz_row"], 0.1)
        L, R = _unit_columns(g, m, 4, 1.0), _unit_columns(g, n, 4, 1.0)
        st.op = pg.CsrOperator(S, L, R, 50.0 * 0.85 ** np.arange(4))
        st.model = pg_learned.StartModel(seed=seed)
        Q = torch.linalg.qr(torch.randn(m, k, generator=g, device="cuda", dtype=torch.float64))[0]
        st.U = np.asfortranarray(Q.cpu().numpy())
        return st
    if kind == "apply":
        S = _apply_matrix(case, seed)
        st.op = pg.CsrOperator(S)
        m, n = S.shape
        st.x, st.xt = (torch.from_numpy(_start(seed + j, d)).cuda() for j, d in ((0, n), (1, m)))
        st.y, st.yt = (torch.empty(d, dtype=torch.float64, device="cuda") for d in (m, n))
        torch.cuda.synchronize()
        return st
    S, L, R, w = _matrix(case, seed)
    m, n = S.shape
    st.v0 = _start(seed, m, cplx=kind == "complex")
    if kind == "svdp":
        st.A = S
        return st
    st.op = pg.CsrOperator(S, L, R, w)
    k, kmax = case["k"], case["kmax"]
    if kind != "lansvd":
        # the driver's arrays as the caller keeps them between solves; where the results are large, a caller
        # has the columns that receive them page-locked
        typ = {"single": np.float32, "complex": np.complex128}.get(kind, np.float64)
        st.U, st.V = _array(m, kmax + 1, typ), _array(n, kmax, typ)
        if kind in ("zipf", "complex"):
            st.locked = [_Locked(st.U[:, :k]), _Locked(st.V[:, :k])]
    return st


def _apply_matrix(case, seed):
    """Row lengths 1 + Poisson(mean - 1), uniform columns."""
    g = _gen(seed)
    m, n = case["m"], case["n"]
    cnt = 1 + torch.poisson(torch.full((m,), case["mean"] - 1.0, device="cuda"), generator=g).to(torch.int64)
    nnz = int(cnt.sum())
    ptr = np.zeros(m + 1, dtype=np.int64)
    np.cumsum(cnt.cpu().numpy(), out=ptr[1:])
    idx = torch.randint(0, n, (nnz,), generator=g, device="cuda", dtype=torch.int32)
    val = torch.randn(nnz, generator=g, device="cuda", dtype=torch.float64)
    return sp.csr_array((val.cpu().numpy(), idx.cpu().numpy(), ptr), shape=(m, n))


# --------------------------------------------------------------------- run
def run(st):
    kind = st.case["kind"]
    return {"lansvd": _run_lansvd, "svdp": _run_svdp, "factored": _run_irl, "zipf": _run_irl, "single": _run_single,
            "complex": _run_complex, "batch": _run_batch, "learned": _run_learned, "apply": _run_apply}[kind](st)


# The error bounds that the drivers return beside the triplets are rounding
# noise at these tolerances; a caller tests them against the tolerance, so
# that test is what goes out.
def _certified(bnd, sigma, tol):
    return bnd <= max(tol, 16 * 2.0 ** -53) * sigma


# A singular pair is determined up to a common sign; as a caller who stores or
# compares the vectors does, each pair is brought to one sign in place: the
# leading entries of its left vector have a sum with a non-negative real part
# (complex pairs: the start vector fixes all of their phase but the sign).
def _one_sign(ut, vt):
    """ut (k x m) and vt (k x n): torch views of the left and right vectors, one per row."""
    for j, lead in enumerate(ut[:, :1000].sum(dim=1).tolist()):
        if (lead.real if isinstance(lead, complex) else lead) < 0:
            ut[j].neg_()
            vt[j].neg_()


def _run_lansvd(st):
    c = st.case
    u, s, vt, bnd = pg.svdp(st.op, c["k"], irl_mode=False, kmax=c["kmax"], tol=_tol(c), v0=st.v0,
                            rng=np.random.default_rng(0))
    _one_sign(torch.from_numpy(u.T), torch.from_numpy(vt))
    return {"u": u, "s": s, "vt": vt, "ok": _certified(bnd, s, _tol(c))}


def _run_svdp(st):
    c = st.case
    u, s, vt, bnd = pg.svdp(st.A, c["k"], kmax=c["kmax"], tol=_tol(c), v0=st.v0, rng=np.random.default_rng(0))
    _one_sign(torch.from_numpy(u.T), torch.from_numpy(vt))
    return {"u": u, "s": s, "vt": vt, "ok": _certified(bnd, s, _tol(c))}


_DOPT = (math.sqrt(2.0 ** -52), (2.0 ** -52) ** 0.75, 0.0, 0.002)


def _run_irl(st):
    c = st.case
    m, n = st.op.shape
    k, dim = c["k"], c["kmax"]
    sigma, bnd = np.zeros(k), np.zeros(k)
    st.U[:, 0] = st.v0
    pg.set_precision(c.get("precision", "fp64"))
    try:
        kc, info = pg.lansvd_irl(b"L", b"y", b"y", m, n, dim, dim - k, k, 100, st.op.aprod, st.U, sigma, bnd, st.V,
                                 _tol(c), np.array(_DOPT), np.array((0, 1), dtype=np.int32), iparm=st.op.iparm)
    finally:
        pg.set_precision("fp64")
    _one_sign(torch.from_numpy(st.U.T[:k]), torch.from_numpy(st.V.T[:k]))
    return {"u": st.U[:, :k], "s": sigma, "v": st.V[:, :k], "converged": kc, "info": info}


def _run_complex(st):
    c = st.case
    m, n = st.op.shape
    k, dim = c["k"], c["kmax"]
    sigma, bnd = np.zeros(k), np.zeros(k)
    st.U[:, 0] = st.v0
    kc, info = pg.zlansvd_irl(b"L", b"y", b"y", m, n, dim, dim - k, k, 100, st.op.aprod, st.U, sigma, bnd, st.V,
                              _tol(c), np.array(_DOPT), np.array((0, 1), dtype=np.int32), iparm=st.op.iparm)
    _one_sign(torch.from_numpy(st.U.T[:k]), torch.from_numpy(st.V.T[:k]))
    return {"u": st.U[:, :k], "s": sigma, "v": st.V[:, :k], "converged": kc, "info": info}


def _run_single(st):
    c = st.case
    m, n = st.op.shape
    k, dim = c["k"], c["kmax"]
    lib = pg.load()
    ci = lambda v: C.byref(C.c_int(v))  # noqa: E731
    p = lambda a: C.c_void_p(a.ctypes.data)  # noqa: E731
    lwork, liwork, _ = pg.work_sizes(m, n, dim)
    work, iwork = np.empty(lwork, dtype=np.float32), np.empty(liwork, dtype=np.int32)
    sigma, bnd = np.zeros(k, dtype=np.float32), np.zeros(k, dtype=np.float32)
    eps = 2.0 ** -23
    dopt = np.array((math.sqrt(eps), eps ** 0.75, 0.0, 0.002), dtype=np.float32)
    iopt, dparm = np.array((0, 1), dtype=np.int32), np.zeros(1, dtype=np.float32)
    ne, info = C.c_int(k), C.c_int(0)
    st.U[:, 0] = st.v0
    lib.slansvd_irl_(b"L", b"y", b"y", ci(m), ci(n), ci(dim), ci(dim - k), C.byref(ne), ci(100),
                     lib.propack_gpu_csr_saprod_, p(st.U), ci(m), p(sigma), p(bnd), p(st.V), ci(n),
                     C.byref(C.c_float(_tol(c))), p(work), ci(lwork), p(iwork), ci(liwork), p(dopt), p(iopt),
                     C.byref(info), p(dparm), p(st.op.iparm), C.c_size_t(1), C.c_size_t(1), C.c_size_t(1))
    _one_sign(torch.from_numpy(st.U.T[:k]), torch.from_numpy(st.V.T[:k]))
    return {"u": st.U[:, :k], "s": sigma, "v": st.V[:, :k], "converged": ne.value, "info": info.value}


def _run_batch(st):
    c, b = st.case, st.batch
    dp = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731
    rc = pg.load().propack_batch_solve(b.handle, c["kmax"], c["k"], 100, _tol(c), dp(st.u0), dp(st.sigma),
                                       dp(st.bnd), st.info.ctypes.data_as(C.POINTER(C.c_int)), dp(st.U), dp(st.V))
    if rc != 0:
        raise pg.PropackError(f"propack_batch_solve failed ({rc}): {pg.last_error()}")
    k = c["k"]
    ut = torch.from_numpy(st.U).split([k * int(m) for m in b.m])
    vt = torch.from_numpy(st.V).split([k * int(n) for n in b.n])
    for u, v in zip(ut, vt):
        u, v = u.view(k, -1), v.view(k, -1)
        sign = torch.where(u[:, :1000].sum(dim=1, keepdim=True) < 0, -1.0, 1.0)
        u.mul_(sign)
        v.mul_(sign)
    return {"s": st.sigma, "info": st.info, "u": st.U, "v": st.V}


def _run_learned(st):
    if st.case["grad"]:
        loss, grad = st.model.grad(st.op, st.U)
        return {"loss": loss, "grad": grad}
    return {"u0": st.model.start(st.op)}


def _run_apply(st):
    lib = pg.load()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for trans, x, y in ((0, st.x, st.y), (1, st.xt, st.yt)):
        rc = lib.propack_csr_apply_noalloc(C.c_int64(st.op.handle), C.c_int(trans), C.c_void_p(x.data_ptr()),
                                           C.c_void_p(y.data_ptr()), stream)
        if rc != 0:
            raise pg.PropackError(f"propack_csr_apply_noalloc failed ({rc}): {pg.last_error()}")
    return {"y": st.y, "yt": st.yt}


# -------------------------------------------------------------------- work
def work(case):
    """Input read once and output written once.  A solver cannot do with fewer than k steps of the two products
    and the k columns of U and V kept orthogonal, each column read once per later step on its side."""
    kind = case["kind"]
    if kind == "batch":
        m, n, k, p = 10_250.0, 4100.0, case["k"], case["nprob"]
        nnz = 0.01 * m * n
        return {"bytes": p * (k * 2 * nnz * 8 + k * k * (m + n) * 8 / 2 + 2 * k * (m + n) * 8),
                "flops": p * (k * 4 * nnz + 2 * k * k * (m + n))}
    if kind == "learned":
        m, nnz, k = case["m"], case["m"] * case["nnz_row"], case["k"]
        flops = 2.0 * m * (18 * 256 + 256 * 256 + 256)
        if case["grad"]:
            return {"bytes": nnz * 12.0 + m * (8.0 * k + 72), "flops": 3 * flops}
        return {"bytes": nnz * 12.0 + m * 80.0, "flops": flops}
    if kind == "apply":
        nnz = case["m"] * case["mean"]
        return {"bytes": 2 * (12.0 * nnz + 8.0 * (case["m"] + case["n"]) + 4.0 * case["m"]), "flops": 4.0 * nnz}
    k = case["k"]
    m, n = case["m"], case.get("n", case["m"])
    es = {"single": 4, "complex": 16}.get(kind, 8)
    nnz = m * case["nnz_row"] if "nnz_row" in case else 7.75 * m
    if kind == "factored":
        nnz += case["rank"] * (case["udens"] * m + case["vdens"] * n)
    fl = 4 if kind == "complex" else 1
    return {"bytes": 2 * k * nnz * (es + 4) + es * (m + n) * (k * k / 2 + 4 * k),
            "flops": fl * (4 * k * nnz + 2 * k * k * (m + n))}


# ------------------------------------------------------------------- exact
def _lanczos_values(mv, rmv, m, n, k, dim, v0, dtype):
    """The k largest singular values by dim steps of Golub-Kahan Lanczos with full reorthogonalisation in 64 bits
    (dim <= min(m, n); the leading values have converged to rounding well before)."""
    U = torch.empty(dim, m, dtype=dtype, device="cuda")
    V = torch.empty(dim, n, dtype=dtype, device="cuda")
    B = np.zeros((dim + 1, dim))
    u = v0 / v0.norm()
    for j in range(dim):
        U[j] = u
        v = rmv(u)
        for _ in range(2):
            v = v - (V[:j].conj() @ v) @ V[:j]
        B[j, j] = float(v.norm())
        v = v / B[j, j]
        V[j] = v
        u = mv(v)
        for _ in range(2):
            u = u - (U[:j + 1].conj() @ u) @ U[:j + 1]
        B[j + 1, j] = float(u.norm())
        u = u / B[j + 1, j]
    return np.linalg.svd(B, compute_uv=False)[:k]


def _sparse(A):
    A = sp.csr_array(A)
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=d)).cuda()  # noqa: E731
    val = t(A.data, A.data.dtype)
    fwd = torch.sparse_csr_tensor(t(A.indptr, np.int64), t(A.indices, np.int64), val, size=A.shape)
    At = A.conj().T.tocsr()
    adj = torch.sparse_csr_tensor(t(At.indptr, np.int64), t(At.indices, np.int64), t(At.data, At.data.dtype),
                                  size=At.shape)
    return (lambda x: fwd @ x), (lambda x: adj @ x)


def exact(case, seed):
    """The singular values (the vectors are determined up to their signs only) or the products in 64 bits."""
    kind = case["kind"]
    if kind == "learned":
        return None  # its sketch and its weights are drawn inside the library
    if kind == "apply":
        S = _apply_matrix(case, seed)
        m, n = S.shape
        return {"y": S @ _start(seed, n), "yt": S.T @ _start(seed + 1, m)}
    if kind == "batch":
        k, out = case["k"], []
        if case["nprob"] > 256:
            return None
        for A in _batch_mats(case, seed):
            mv, rmv = _sparse(A)
            g = _gen(seed)
            v0 = torch.rand(A.shape[0], generator=g, device="cuda", dtype=torch.float64)
            out.append(_lanczos_values(mv, rmv, *A.shape, k, min(64, *A.shape), v0, torch.float64))
        return {"s": np.array(out), "info": None, "u": None, "v": None}
    S, L, R, w = _matrix(case, seed)
    m, n = S.shape
    typ = torch.complex128 if kind == "complex" else torch.float64
    mv0, rmv0 = _sparse(S)
    mv, rmv = mv0, rmv0
    if L is not None:
        (lm, lr), (rm, rr) = _sparse(L), _sparse(R)
        wt = torch.from_numpy(w).cuda()
        mv = lambda x: mv0(x) + lm(wt * rr(x))  # noqa: E731
        rmv = lambda x: rmv0(x) + rm(wt * lr(x))  # noqa: E731
    v0 = torch.from_numpy(_start(seed, m, cplx=kind == "complex")).cuda()
    dim = min(m, n, max(3 * case["k"] + 40, 200))
    s = _lanczos_values(mv, rmv, m, n, case["k"], dim, v0, typ)
    if kind in ("lansvd", "svdp"):
        return {"u": None, "s": s, "vt": None, "ok": None}
    s = s.astype(np.float32).astype(np.float64) if kind == "single" else s
    return {"u": None, "s": s, "v": None, "converged": None, "info": None}
