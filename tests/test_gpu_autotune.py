"""Autotuning leaves every layout of the handle on the chosen slab geometry, and
a small FP64 system on the kernels of small systems."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("maker", ["poisson2d_60", "varpoisson3d_40"])
def test_set_precisions_layout_follows_the_tuned_geometry(mf, maker):
    """The layout of mf_tiles_set_precisions shares the copy ring's stages with the FP64 layout."""
    import torch

    kind, size = maker.rsplit("_", 1)
    A = mf.Matrix.poisson2d(int(size)) if kind == "poisson2d" else mf.Matrix.varpoisson3d(int(size), 0.1, 10.0, seed=5)
    t = mf.Tiles(A)
    prec = np.random.default_rng(1).choice([mf.PREC_FP64, mf.PREC_FP32], t.info()["tilenum"]).astype(np.uint8)
    t.set_precisions(prec)
    x = torch.tensor(np.random.default_rng(2).standard_normal(A.n), device="cuda")
    y0, y1 = torch.empty_like(x), torch.empty_like(x)
    t.spmv_level_dev(0, x.data_ptr(), y0.data_ptr())
    for _ in range(2):
        t.autotune(reps=3)
        t.spmv_level_dev(0, x.data_ptr(), y1.data_ptr())
        assert torch.equal(y0, y1)
    assert np.array_equal(t.precisions()[0], prec)
    _, r = t.solve_cg(A.b(), tol=1e-10, maxiter=20000, opts=mf.options(precision_mode=mf.MODE_MIXED_RULE))
    assert r["status"] == 0 and r["iters_level"][0] > 0 and r["rel_residual_true"] <= 1.5e-10


def _vector_bytes(res, n, spmvs):
    """Vector bytes a row and iteration of the kernel that ran, from the result's byte count."""
    per = (res["total_bytes"] - res["spmv_bytes_fp64"] - 16.0 * n) / res["iterations"]
    return (per - spmvs * res["spmv_bytes_fp64"]) / n


@pytest.mark.parametrize("maker", ["poisson2d_37", "poisson2d_120", "varpoisson3d_20", "varpoisson3d_36"])
def test_tuned_small_systems_stay_on_the_resident_kernels(mf, maker):
    kind, size = maker.rsplit("_", 1)
    A = mf.Matrix.poisson2d(int(size)) if kind == "poisson2d" else mf.Matrix.varpoisson3d(int(size), 0.1, 10.0, seed=5)
    t = mf.Tiles(A)
    few = t.info()["nctas"]
    assert few < 148
    t.autotune(reps=3)
    info = t.info()
    # few CTAs with one slab each, or every SM where the tuned slabs are smaller than that
    assert (info["nctas"], info["nslabs"]) == (few, few) or info["nctas"] == 148
    for solve, spmvs, vec in ((t.solve_cg, 1, 8.0), (t.solve_pcg, 1, 8.0), (t.solve_bicgstab, 2, 16.0)):
        _, r = solve(A.b(), tol=1e-10, maxiter=20000)
        assert r["status"] == 0 and r["rel_residual_true"] <= 1.5e-10
        assert _vector_bytes(r, A.n, spmvs) == pytest.approx(vec, abs=1e-6)
