"""The group-wide sums add the CTAs' shares in one fixed order, whatever polls
them: rank c goes to lane c mod 32 in ascending c, then a xor tree over the 32
lanes. Diagonal systems with one nonzero residual entry a CTA, whose shares are
exact, show that order to the bit: in the first step of the CG (x there is
r.r / d.Ad), in the residual before the first step, and in the mixed CG's four
values of one sum."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ordered(p):
    lanes = [0.0] * 32
    for c, v in enumerate(p):
        lanes[c % 32] += float(v)
    for o in (16, 8, 4, 2, 1):
        lanes = [lanes[i] + lanes[i ^ o] for i in range(32)]
    return lanes[0]


def _values(G, seed):
    """One residual entry a CTA, 1 in CTA 0: 24-bit values, so that FP32 holds them and their squares are exact."""
    rng = np.random.default_rng(seed)
    r = np.ldexp(rng.integers(1 << 23, 1 << 24, G).astype(np.float64), rng.integers(-33, -15, G))
    r[0] = 1.0
    return r


def _diag(n, rows, a):
    d = np.ones(n)
    d[rows] = a
    return np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d


# the CTAs of small FP64 systems (28 row blocks each), and every SM
CTAS = [16, 31, 33, 64, 97, 111, 148]


def _system(mf, G, seed, opts=None):
    per = 30 if G == 148 else 28
    n = 16 * per * G
    rows = 16 * per * np.arange(G)
    a = np.ldexp(1.0, np.random.default_rng(seed).integers(-6, 7, G))
    t = mf.Tiles(csr=(n, n, *_diag(n, rows, a)), opts=opts)
    assert t.info()["nctas"] == G
    return t, n, rows, a


@pytest.mark.parametrize("G", CTAS)
@pytest.mark.parametrize("glob", [0, 1])
def test_cg_first_step(mf, G, glob):
    t, n, rows, a = _system(mf, G, G)
    r = _values(G, G + 1)
    b = np.zeros(n)
    b[rows] = r
    o = mf.options(fixed_iterations=1)
    o.reserved[5] = glob
    x, _ = t.solve_cg(b, tol=1e-300, maxiter=1, opts=o)
    assert x[0] == _ordered(r * r) / _ordered(r * (a * r))


@pytest.mark.parametrize("G", CTAS)
@pytest.mark.parametrize("solver", ["solve_cg", "solve_pcg", "solve_bicgstab"])
@pytest.mark.parametrize("glob", [0, 1])
def test_residual_before_the_first_step(mf, G, solver, glob):
    t, n, rows, a = _system(mf, G, G)
    r = _values(G, G + 2)
    b, x0 = np.zeros(n), np.zeros(n)
    b[0] = 1.0  # b.b = 1
    x0[rows[1:]] = -r[1:] / a[1:]
    o = mf.options()
    o.reserved[5] = glob
    _, res = getattr(t, solver)(b, x0=x0, tol=1e-300, maxiter=0, opts=o)
    assert res["rel_residual_rec"] == math.sqrt(_ordered(r * r))


@pytest.mark.parametrize("glob", [0, 1])
def test_mixed_cg_sum_of_four(mf, glob):
    G = 148
    t, n, rows, a = _system(mf, G, 5, mf.options(precision_mode=mf.MODE_FIXED, fixed_precision=mf.PREC_FP32))
    r = _values(G, 6)
    b, x0 = np.zeros(n), np.zeros(n)
    b[0] = 1.0
    x0[rows[1:]] = -r[1:] / a[1:]
    o = mf.options(precision_mode=mf.MODE_FIXED, fixed_precision=mf.PREC_FP32)
    o.reserved[5] = glob
    _, res = t.solve_cg(b, x0=x0, tol=1e-300, maxiter=1, opts=o)
    assert res["iters_level"][0] == 1
    rel = math.sqrt(_ordered(r * r))
    assert res["rel_residual_rec"] == math.sqrt(rel * rel)


@pytest.mark.parametrize("gs", [1, 31, 32, 33, 65, 97, 128, 129, 148])
def test_batched_cg_first_step(mf, gs):
    import torch

    n = 16 * 3 * gs
    rows = 48 * np.arange(gs)
    a = np.ldexp(1.0, np.random.default_rng(gs).integers(-6, 7, gs))
    r = _values(gs, gs + 3)
    bh = np.zeros(n)
    bh[rows] = r
    o = mf.options(fixed_iterations=1)
    o.reserved[4] = gs
    B = mf.Batch([mf.Matrix.from_csr(n, n, *_diag(n, rows, a))], o)
    b = torch.tensor(bh, device="cuda")
    x = torch.zeros_like(b)
    B.solve_cg_dev(b.data_ptr(), x.data_ptr(), 1e-300, 1)
    assert float(x[0]) == _ordered(r * r) / _ordered(r * (a * r))
