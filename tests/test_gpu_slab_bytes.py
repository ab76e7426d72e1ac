"""The largest slab_bytes that fits: 4 stages of 41472 + 14464 bytes leave 8704
of the 232448 bytes of shared memory a CTA may have for a kernel's own arrays
(the mixed tensor-memory CG needs most)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_largest_slab_bytes_is_accepted(mf, O):
    A = mf.Matrix.varpoisson3d(20, 0.1, 10.0, seed=3)
    rp, ci, v = A.csr()
    b = A.b()
    o = O.OracleTiles(A.n, A.n, rp, ci, v)
    for mode in (mf.MODE_FP64, mf.MODE_MIXED_RULE):
        t = mf.Tiles(A, mf.options(slab_bytes=41472, precision_mode=mode))
        assert np.array_equal(t.spmv(b), o.spmv(b))
        for solve in (t.solve_cg, t.solve_pcg, t.solve_bicgstab):
            _, r = solve(b, tol=1e-10, maxiter=5000)
            assert r["status"] == 0 and r["rel_residual_true"] <= 1.5e-10


def test_larger_slab_bytes_is_refused(mf):
    with pytest.raises(mf.MfError):
        mf.Tiles(mf.Matrix.poisson2d(20), mf.options(slab_bytes=41984))
