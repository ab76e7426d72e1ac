"""A handle keeps working after another one was encoded or tuned with smaller slabs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [20, 60])  # resident kernels, tensor-memory kernels
@pytest.mark.parametrize("other", ["encode", "autotune"])
def test_other_handles_slab_size(mf, size, other):
    A = mf.Matrix.varpoisson3d(size, 0.1, 10.0, seed=5)
    t = mf.Tiles(A)
    x = np.random.default_rng(2).standard_normal(A.n)

    def results():
        out = [t.spmv(x)]
        for name in ("solve_cg", "solve_pcg", "solve_bicgstab"):
            sol, r = getattr(t, name)(A.b(), tol=1e-10, maxiter=20000)
            assert r["status"] == 0
            out.append(sol)
        return out

    before = results()
    B = mf.Matrix.poisson2d(40)
    small = mf.Tiles(B, opts=mf.options(slab_bytes=24576))
    if other == "autotune":
        small.autotune(reps=1)
    small2 = mf.Tiles(B, opts=mf.options(slab_bytes=16384))
    for u, v in zip(before, results()):
        assert np.array_equal(u, v)
    assert small2.solve_cg(B.b(), tol=1e-10)[1]["status"] == 0
