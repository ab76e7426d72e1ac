"""A wait that runs out inside an iteration of the resident kernels (their
producer warp waits for an epoch that no CTA publishes) ends the solve after
one time limit, not one for the producer and another for the consumers, and
leaves the context and the handle usable."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 0.5


@pytest.mark.parametrize("solver", ["solve_cg", "solve_pcg", "solve_bicgstab"])
@pytest.mark.parametrize("N", [20, 300])  # one slab on few CTAs; two slabs on every SM
def test_wait_in_an_iteration_ends_after_one_limit(mf, solver, N):
    A = mf.Matrix.poisson2d(N)
    t = mf.Tiles(A)
    solve = getattr(t, solver)
    b = A.b()
    x, before = solve(b, tol=1e-10)
    assert before["status"] == 0
    o = mf.options(timeout_s=LIMIT)
    o.reserved[0] = 0x5742
    t0 = time.perf_counter()
    with pytest.raises(mf.MfError) as e:
        solve(b, tol=1e-10, opts=o)
    spent = time.perf_counter() - t0
    assert e.value.status == mf.MF_ERR_TIMEOUT
    assert LIMIT <= spent < 1.5 * LIMIT
    x2, after = solve(b, tol=1e-10)
    assert after["status"] == 0 and after["iterations"] == before["iterations"] and np.array_equal(x, x2)
