"""Precisions set on a small FP64 handle run on the grid of a mixed handle: the
rounding of the grid sums, which mixed solves decide on, follows the CTA count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("maker", ["poisson2d_37", "poisson2d_222", "varpoisson3d_13", "varpoisson3d_36"])
@pytest.mark.parametrize("tuned", [False, True])
def test_mixed_solves_equal_a_mixed_handles(mf, maker, tuned):
    kind, size = maker.rsplit("_", 1)
    A = mf.Matrix.poisson2d(int(size)) if kind == "poisson2d" else mf.Matrix.varpoisson3d(int(size), 0.1, 10.0, seed=5)
    mixed = mf.options(precision_mode=mf.MODE_MIXED_RULE)
    ref, t = mf.Tiles(A, opts=mixed), mf.Tiles(A)
    few, every = t.info()["nctas"], ref.info()["nctas"]
    assert few < every
    prec = np.random.default_rng(1).choice([mf.PREC_FP64, mf.PREC_FP32], t.info()["tilenum"]).astype(np.uint8)
    x = np.random.default_rng(2).standard_normal(A.n)
    y = t.spmv(x)
    ref.set_precisions(prec)
    t.set_precisions(prec)
    assert t.info()["nctas"] == every
    if tuned:  # another slab geometry may stay, the grid does not shrink again
        t.autotune(reps=3)
        assert t.info()["nctas"] == every
    assert np.array_equal(t.spmv(x), y)
    for name in ("solve_cg", "solve_bicgstab", "solve_pcg"):
        xr, r = getattr(ref, name)(A.b(), tol=1e-10, maxiter=20000, opts=mixed)
        xt, q = getattr(t, name)(A.b(), tol=1e-10, maxiter=20000, opts=mixed)
        assert r["status"] == q["status"] == 0
        if not tuned:  # the CTAs' row ranges are the same
            assert r["iterations"] == q["iterations"]
            assert np.array_equal(xr, xt)
