"""Every kernel a system can be sent to, at the sizes where it can go wrong:
tiny, ragged and empty CTA ranges, b = 0, maxiter = 0, a wait that runs out.
reserved[5] chooses the route: 0 the library's choice (small systems: matrix
in shared memory, vectors in registers; scattered ones: direct gathers), 2 the
tensor-memory kernels of large systems, 1 the global-vector kernels. The
result's byte count tells which kernel ran."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# vector bytes a row and iteration (mf_result.total_bytes)
BYTES = {"solve_cg": {0: 8, 2: 32, 1: 56}, "solve_pcg": {0: 8, 2: 40, 1: 72},
         "solve_bicgstab": {0: 16, 2: 112, 1: 112}}
DIRECT = 56  # CG by direct gathers


def _vector_bytes(res, n, spmvs=1):
    per = (res["total_bytes"] - res["spmv_bytes_fp64"] - 16.0 * n) / res["iterations"]
    return (per - spmvs * res["spmv_bytes_fp64"]) / n


def _opts(mf, route, **kw):
    o = mf.options(**kw)
    o.reserved[5] = route
    return o


def _tridiag(n, lo=-1.0, d=2.5, hi=-1.0):
    import scipy.sparse as sp

    M = sp.diags([np.full(n - 1, lo), np.full(n, d), np.full(n - 1, hi)], [-1, 0, 1], format="csr")
    M.sort_indices()
    return M


@pytest.mark.parametrize("route", [0, 2, 1])
@pytest.mark.parametrize("n", [1, 5, 16, 17, 33, 2047])
def test_tiny_and_ragged_systems(mf, O, n, route):
    b = np.random.default_rng(n).uniform(-1, 1, n)
    for solver, lo, hi in (("solve_cg", -1.0, -1.0), ("solve_pcg", -1.0, -1.0), ("solve_bicgstab", -1.3, -0.7)):
        M = _tridiag(n, lo, 2.5, hi)
        csr = (M.indptr.astype(np.int32), M.indices.astype(np.int32), M.data)
        t = mf.Tiles(csr=(n, n, *csr))
        x, r = getattr(t, solver)(b, tol=1e-10, maxiter=1000, opts=_opts(mf, route))
        assert r["status"] == 0 and np.linalg.norm(b - M @ x) / np.linalg.norm(b) <= 2e-10, (solver, r)
        assert _vector_bytes(r, n, 2 if solver == "solve_bicgstab" else 1) == pytest.approx(BYTES[solver][route], abs=1e-6)
        if n % 16 == 1 or solver == "solve_pcg":
            continue  # Tile_create stores no values for a 1-row tail block: the oracle's matrix is another one
        o = O.OracleTiles(n, n, *csr)
        it_o = (o.cg if solver == "solve_cg" else o.bicgstab)(b, 1e-10, 1000)[0]
        assert abs(r["iterations"] - it_o) <= 2, (solver, r, it_o)


@pytest.mark.parametrize("route", [0, 2, 1])
def test_zero_rhs_and_zero_maxiter(mf, route):
    A = mf.Matrix.poisson2d(32)
    t = mf.Tiles(A)
    o = _opts(mf, route)
    for solve in (t.solve_cg, t.solve_bicgstab, t.solve_pcg):
        x, r = solve(np.zeros(A.n), tol=1e-10, maxiter=100, opts=o)
        assert r["status"] == 0 and r["iterations"] == 0 and not x.any()
        x0 = np.full(A.n, 0.5)
        x, r = solve(A.b(), x0=x0, tol=1e-10, maxiter=0, opts=o)
        assert r["status"] == mf.MF_ERR_NOT_CONVERGED and r["iterations"] == 0 and np.array_equal(x, x0)


@pytest.mark.parametrize("route", [0, 2, 1])
@pytest.mark.parametrize("scattered", [False, True])
def test_bounded_wait(mf, route, scattered):
    A = mf.Matrix.spd_random(12000, 5) if scattered else mf.Matrix.poisson2d(64)
    t = mf.Tiles(A)
    o = _opts(mf, route, timeout_s=0.05)
    o.reserved[0] = 0x5741
    with pytest.raises(mf.MfError) as e:
        t.solve_cg(A.b(), opts=o)
    assert e.value.status == mf.MF_ERR_TIMEOUT
    _, r = t.solve_cg(A.b(), tol=1e-10, opts=_opts(mf, route))
    assert r["status"] == 0


@pytest.mark.parametrize("maker", ["varpoisson3d_24", "spd_random_30000"])
def test_noalloc_against_every_route(mf, maker):
    import torch

    kind, size = maker.rsplit("_", 1)
    A = mf.Matrix.varpoisson3d(int(size)) if kind == "varpoisson3d" else mf.Matrix.spd_random(int(size), 9)
    t = mf.Tiles(A)
    b = torch.tensor(A.b(), device="cuda")
    x = torch.zeros_like(b)
    res = mf.MfResult()
    o = mf.options(check_true_residual=1)
    rc = mf.lib().mf_solve_cg_dev_noalloc(t.h, C.c_void_p(b.data_ptr()), C.c_void_p(x.data_ptr()), 1e-10, 20000,
                                          C.byref(o), C.byref(res))
    na, ran = res.as_dict(), []
    assert rc == 0 and na["rel_residual_true"] <= 1.1e-10
    for route in (0, 2, 1):
        _, r = t.solve_cg(A.b(), tol=1e-10, maxiter=20000, opts=_opts(mf, route))
        assert r["status"] == 0 and abs(r["iterations"] - na["iterations"]) <= max(2, 0.02 * na["iterations"])
        ran.append(round(_vector_bytes(r, A.n)))
    assert ran == ([8, 32, 56] if kind == "varpoisson3d" else [DIRECT, 32, DIRECT])


# rows of 1..9 entries (around the 8 gathers a lane keeps in flight) and of 4..40, empty row blocks at either end
@pytest.mark.parametrize("n,lo,hi,empty", [(8007, 1, 9, []), (12000, 4, 40, [(0, 16), (11984, 12000)]),
                                           (9001, 0, 20, [(3200, 3264)])])
def test_direct_spmv_runs_and_is_bitexact(mf, O, n, lo, hi, empty):
    rng = np.random.default_rng(n)
    lens = rng.integers(lo, hi + 1, n)
    for a, e in empty:
        lens[a:e] = 0
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in lens]).astype(np.int32)
    v = rng.standard_normal(len(ci))
    t = mf.Tiles(csr=(n, n, rp, ci, v))
    o = O.OracleTiles(n, n, rp, ci, v)
    b = rng.standard_normal(n)
    _, r = t.solve_cg(b, tol=1e-300, maxiter=1, opts=mf.options(fixed_iterations=1))
    assert r["iterations"] == 1 and round(_vector_bytes(r, n)) == DIRECT  # the handle's layout is direct
    for x in (b, np.where(rng.random(n) < 0.01, np.inf, b)):
        y, yo = t.spmv(x), o.spmv(x)
        if n % 16 == 1:  # the oracle's tail block has no values
            y, yo = y[:-1], yo[:-1]
        assert np.array_equal(y, yo, equal_nan=True)


@pytest.mark.parametrize("route", [0, 2])
@pytest.mark.parametrize("n", [6000, 30008])
def test_scattered_cg_matches_oracle(mf, O, n, route):
    A = mf.Matrix.spd_random(n, 11)
    b = A.b()
    x, r = mf.Tiles(A).solve_cg(b, tol=1e-10, maxiter=5000, opts=_opts(mf, route))
    it_o, x_o, _ = O.OracleTiles(n, n, *A.csr()).cg(b, 1e-10, 5000)
    assert round(_vector_bytes(r, n)) == (DIRECT if route == 0 else 32)
    assert r["status"] == 0 and r["rel_residual_true"] <= 1.5e-10
    assert abs(r["iterations"] - it_o) <= max(2, 0.02 * it_o)
    assert np.linalg.norm(x - x_o) / np.linalg.norm(x_o) < 1e-7
