"""Sums of at most 32 CTAs run in kernels of their own, one warp a value: the
order at the edge, and the sum of four values."""
import numpy as np
import pytest
from test_gpu_sum_order import _ordered, _system, _values

pytestmark = pytest.mark.gpu


def test_first_step_on_32_ctas(mf):
    t, n, rows, a = _system(mf, 32, 32)
    r = _values(32, 7)
    b = np.zeros(n)
    b[rows] = r
    for solve in (t.solve_cg, t.solve_pcg):
        x, _ = solve(b, tol=1e-300, maxiter=1, opts=mf.options(fixed_iterations=1))
        if solve == t.solve_cg:
            assert x[0] == _ordered(r * r) / _ordered(r * (a * r))
        else:
            assert np.allclose(x[rows] * a, r, rtol=1e-14, atol=0)  # a diagonal system: one step


@pytest.mark.parametrize("G", [16, 31, 32, 33])
def test_bicgstab_first_step(mf, G):
    """x = alpha p + omega s with t.s and t.t from the sum of four values."""
    t, n, rows, a = _system(mf, G, G)
    r = _values(G, G + 4)
    b = np.zeros(n)
    b[rows] = r
    x, _ = t.solve_bicgstab(b, tol=1e-300, maxiter=1, opts=mf.options(fixed_iterations=1))
    alpha = _ordered(r * r) / _ordered(r * (a * r))
    s = r - alpha * (a * r)
    omega = _ordered(a * s * s) / _ordered(a * s * (a * s))
    # a handful of roundings, of terms no larger than these
    scale = np.abs(alpha * r) + np.abs(omega) * (np.abs(r) + np.abs(alpha * a * r))
    assert np.all(np.abs(x[rows] - (alpha * r + omega * s)) <= 64 * np.finfo(np.float64).eps * scale)
