"""Direct layouts (scattered matrices: every row block gathers its x entries,
without the copy ring): SpMV bit for bit in the oracle's order, with empty row
blocks at either end, row lengths around the gather batch, ragged tails and
a rectangular matrix; CG on the direct kernel against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scattered(n, ncols, lens, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(ncols, int(k), replace=False)) for k in lens] or [[]]).astype(np.int32)
    return rp, ci, rng.standard_normal(len(ci))


# rows of 0..40 entries over the gather batch of 8, rows not a multiple of 16
@pytest.mark.parametrize("n,ncols,lo,hi,empty", [
    (2010, 2010, 1, 9, []),
    (3007, 3007, 0, 40, [(0, 40), (1600, 1650), (2980, 3007)]),
    (40000, 40000, 6, 18, [(0, 16), (39984, 40000)]),
    (5003, 4008, 3, 17, []),
])
def test_direct_spmv_bitexact(mf, O, n, ncols, lo, hi, empty):
    lens = np.random.default_rng(n).integers(lo, hi + 1, n)
    for a, b in empty:
        lens[a:b] = 0
    rp, ci, v = _scattered(n, ncols, lens, n + 1)
    t = mf.Tiles(csr=(n, ncols, rp, ci, v))
    o = O.OracleTiles(n, ncols, rp, ci, v)
    rng = np.random.default_rng(3)
    for _ in range(2):
        x = rng.standard_normal(ncols) * 10.0 ** rng.uniform(-3, 3, ncols)
        assert np.array_equal(t.spmv(x), o.spmv(x))
    x[7] = np.inf  # infinities and NaN reach the rows that hold them and no others
    x[11] = np.nan
    assert np.array_equal(t.spmv(x), o.spmv(x), equal_nan=True)


@pytest.mark.parametrize("n", [1900, 30008])
def test_direct_cg_matches_oracle(mf, O, n):
    A = mf.Matrix.spd_random(n, 11)
    rp, ci, v = A.csr()
    b = A.b()
    t = mf.Tiles(A)
    x, res = t.solve_cg(b, tol=1e-10, maxiter=5000)
    it_o, x_o, _ = O.OracleTiles(n, n, rp, ci, v).cg(b, 1e-10, 5000)
    assert res["status"] == 0 and res["rel_residual_true"] <= 1.5e-10
    assert abs(res["iterations"] - it_o) <= max(2, 0.02 * it_o)
    assert np.linalg.norm(x - x_o) / np.linalg.norm(x_o) < 1e-7


def test_batch_mixes_small_and_scattered_systems(mf):
    """Systems small enough to be staged by themselves run in a batch that is direct because of the others."""
    import scipy.sparse as sp
    import torch

    mats = [mf.Matrix.spd_random(n, n) for n in (1100, 6000, 16, 9000)] + [mf.Matrix.poisson2d(21)]
    B = mf.Batch(mats)
    b = torch.tensor(np.concatenate([m.b() for m in mats]), device="cuda")
    x = torch.zeros_like(b)
    B.solve_cg_dev(b.data_ptr(), x.data_ptr(), 1e-10, 5000)
    it, st, rel = B.results()
    assert np.all(st == 0) and np.all(rel <= 1e-10)
    xh = x.cpu().numpy()
    for s, m in enumerate(mats):
        rp, ci, v = m.csr()
        M = sp.csr_matrix((v, ci, rp), shape=(m.n, m.n))
        r = m.b() - M @ xh[B.offsets[s]:B.offsets[s + 1]]
        assert np.linalg.norm(r) / np.linalg.norm(m.b()) <= 1.5e-10
