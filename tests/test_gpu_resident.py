"""CG and Jacobi PCG with the matrix in shared memory and the vectors in
registers (small systems), against the global-vector kernels (an option) at
the sizes where a CTA gets its second, third and fourth slab and where the
system no longer fits, and at ragged ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 148 CTAs x 480 rows a slab: 71040, 142080, 213120 and 284160 rows
@pytest.mark.parametrize("kind,size", [("grid2d", 3), ("grid2d", 37), ("grid2d", 266), ("grid2d", 267),
                                       ("grid2d", 377), ("grid2d", 533), ("grid2d", 534), ("grid3d", 41),
                                       ("grid3d", 53), ("grid3d", 63), ("upwind", 20)])
@pytest.mark.parametrize("solver", ["cg", "pcg"])
def test_resident_matches_global_vectors(mf, kind, size, solver):
    if kind == "grid2d":
        A = mf.Matrix.poisson2d(size)
    elif kind == "grid3d":
        A = mf.Matrix.varpoisson3d(size, 0.1, 10.0, seed=3)
    else:
        A = mf.Matrix.convdiff3d(size, v=(0.0, 0.0, 0.0))  # symmetric without a velocity
    n = A.n
    b = np.random.default_rng(size).standard_normal(n)
    x0 = np.random.default_rng(1).standard_normal(n)
    t = mf.Tiles(A)
    o = mf.options()
    o.reserved[5] = 1
    f = t.solve_cg if solver == "cg" else t.solve_pcg
    xg, rg = f(b, x0=x0, tol=1e-10, maxiter=20000, opts=o)
    x, r = f(b, x0=x0, tol=1e-10, maxiter=20000)
    assert rg["status"] == 0 and r["status"] == 0
    assert r["rel_residual_true"] <= 1.5e-10
    assert abs(r["iterations"] - rg["iterations"]) <= max(2, 0.02 * rg["iterations"])
    # the recurrences are the same: after a fixed number of steps only rounding differs
    o.fixed_iterations = 5
    xg, _ = f(b, x0=x0, tol=1e-10, maxiter=20000, opts=o)
    o5 = mf.options(fixed_iterations=5)
    x, r = f(b, x0=x0, tol=1e-10, maxiter=20000, opts=o5)
    assert r["iterations"] == 5
    assert np.linalg.norm(x - xg) <= 1e-12 * np.linalg.norm(xg)


@pytest.mark.parametrize("N", [1, 2, 7, 20, 33, 41, 42, 52, 60, 64])
def test_resident_bicgstab_matches_global_vectors(mf, N):
    A = mf.Matrix.convdiff3d(N)
    b = np.random.default_rng(N).standard_normal(A.n)
    t = mf.Tiles(A)
    o = mf.options()
    o.reserved[5] = 1
    xg, rg = t.solve_bicgstab(b, tol=1e-10, maxiter=2000, opts=o)
    x, r = t.solve_bicgstab(b, tol=1e-10, maxiter=2000)
    assert rg["status"] == 0 and r["status"] == 0
    assert r["rel_residual_true"] <= 1.5e-10
    assert abs(r["iterations"] - rg["iterations"]) <= max(2, 0.02 * rg["iterations"])
    if N > 2:  # (smaller systems are solved exactly before five steps)
        o.fixed_iterations = 5
        xg, _ = t.solve_bicgstab(b, tol=1e-10, maxiter=2000, opts=o)
        x, r = t.solve_bicgstab(b, tol=1e-10, maxiter=2000, opts=mf.options(fixed_iterations=5))
        assert r["iterations"] == 5
        assert np.linalg.norm(x - xg) <= 1e-12 * np.linalg.norm(xg)


# 28 row blocks a CTA, 16 CTAs at least, up to 3/4 of the 148 SMs
@pytest.mark.parametrize("N,ctas", [(4, 16), (84, 16), (85, 17), (222, 111), (224, 148)])
def test_small_systems_take_few_ctas(mf, O, N, ctas):
    A = mf.Matrix.poisson2d(N)
    rp, ci, v = A.csr()
    b = np.random.default_rng(N).standard_normal(A.n)
    t = mf.Tiles(A)
    assert t.info()["nctas"] == ctas
    o = O.OracleTiles(A.n, A.n, rp, ci, v)
    assert np.array_equal(t.spmv(b), o.spmv(b))
    x, r = t.solve_cg(b, tol=1e-10, maxiter=20000)
    it_o, x_o, _ = o.cg(b, 1e-10, 20000)
    assert r["status"] == 0 and r["rel_residual_true"] <= 1.5e-10
    assert abs(r["iterations"] - it_o) <= max(2, 0.02 * it_o)


def test_long_rows_and_mixed_handles_keep_every_sm(mf):
    assert mf.Tiles(mf.Matrix.spd_random(1500, 3)).info()["nctas"] == 148
    t = mf.Tiles(mf.Matrix.poisson2d(60), mf.options(precision_mode=mf.MODE_MIXED_RULE))
    assert t.info()["nctas"] == 148
