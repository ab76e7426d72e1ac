"""The group-wide sums of the persistent solvers (one packet per CTA, polled
32 CTAs a warp) at the edges of their chunks: groups of 1, 31, 32, 33, 65 and
all 148 CTAs, through the batched CG, whose group size is an option."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gs", [1, 31, 32, 33, 65, 148])
def test_group_sums_at_chunk_edges(mf, O, gs):
    import scipy.sparse as sp
    import torch

    mats = [mf.Matrix.spd_random(n, 40 + n) for n in (33, 5000)] + [mf.Matrix.poisson2d(37)]
    o = mf.options()
    o.reserved[4] = gs
    B = mf.Batch(mats, o)
    b = torch.tensor(np.concatenate([m.b() for m in mats]), device="cuda")
    x = torch.zeros_like(b)
    for _ in range(2):  # the second solve starts from the first one's packets
        B.solve_cg_dev(b.data_ptr(), x.data_ptr(), 1e-10, 10000)
    it, st, rel = B.results()
    assert np.all(st == 0) and np.all(rel <= 1e-10)
    xh = x.cpu().numpy()
    for s, m in enumerate(mats):
        rp, ci, v = m.csr()
        M = sp.csr_matrix((v, ci, rp), shape=(m.n, m.n))
        xs = xh[B.offsets[s]:B.offsets[s + 1]]
        assert np.linalg.norm(m.b() - M @ xs) / np.linalg.norm(m.b()) <= 1.5e-10
        if m.n % 16 == 1:
            continue  # Tile_create stores no values for a 1-row tail block: the oracle's CG runs on another matrix
        it_o, _, _ = O.OracleTiles(m.n, m.n, rp, ci, v).cg(m.b(), 1e-10, 10000)
        assert abs(int(it[s]) - it_o) <= max(2, 0.02 * it_o), (s, it[s], it_o)


@pytest.mark.parametrize("sizes", [[16], [40000], [20000, 18, 300], [700] * 40, [3000] + [100] * 150])
def test_batch_default_group_size(mf, sizes):
    """The group size the library chooses: one system, few uneven ones, more systems than groups."""
    import scipy.sparse as sp
    import torch

    mats = [mf.Matrix.spd_random(n, 7 + i) for i, n in enumerate(sizes)]
    B = mf.Batch(mats)
    b = torch.tensor(np.concatenate([m.b() for m in mats]), device="cuda")
    x = torch.zeros_like(b)
    B.solve_cg_dev(b.data_ptr(), x.data_ptr(), 1e-10, 10000)
    it, st, rel = B.results()
    assert np.all(st == 0) and np.all(rel <= 1e-10)
    assert 0 < B.info()["grid"] <= 148
    xh = x.cpu().numpy()
    for s, m in enumerate(mats):
        rp, ci, v = m.csr()
        M = sp.csr_matrix((v, ci, rp), shape=(m.n, m.n))
        r = m.b() - M @ xh[B.offsets[s]:B.offsets[s + 1]]
        assert np.linalg.norm(r) / np.linalg.norm(m.b()) <= 1.5e-10
