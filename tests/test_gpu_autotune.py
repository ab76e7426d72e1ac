"""Autotuning leaves every layout of the handle on the chosen slab geometry."""
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
