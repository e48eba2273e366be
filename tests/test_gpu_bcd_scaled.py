"""FP64 sinkhorn_bcd on the stored plan (csrc/bcd_scaled.cuh) against the FP64
oracle at the edges of its launch shapes: one cluster of 16 blocks up to
65536 entries, a block an SM beyond; fewer rows than blocks or warps, odd
widths, columns split over warps, and regularisations at which the scalings
leave their range so that the base duals move during the solve."""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")

# (n, m, reg, sweeps)
CASES = [
    (1, 7, 0.1, 3), (7, 1, 0.1, 3), (5, 3, 0.05, 20), (16, 65, 0.05, 20), (130, 1, 0.1, 3),
    (3, 1200, 0.05, 20), (1200, 3, 0.05, 20), (256, 256, 0.02, 30), (257, 256, 0.02, 30),
    (151, 701, 0.02, 30), (153, 1030, 0.02, 30), (2000, 35, 0.05, 30), (35, 2001, 0.05, 30),
    (640, 513, 0.01, 30), (180, 140, 0.001, 60), (400, 301, 0.001, 60),
]


@pytest.mark.parametrize("n,m,reg,sweeps", CASES)
def test_scaled_sweeps_follow_the_oracle(n, m, reg, sweeps):
    # The two differ by the rounding of their exponents and sums: z = (alpha +
    # beta - M) / reg is up to 1 / reg in size, so T differs by a few
    # 1e-16 / reg relative, and duals, objectives and marginal errors (of
    # sweeps far from the stop) by that times a small constant.
    M, a, b = erot_points(n, m, seed=n + m, dtype=np.float64)
    r = regot.sinkhorn_bcd(M, a, b, reg, tol=1e-13, max_iter=sweeps)
    o = O.sinkhorn_bcd(M, a, b, reg, tol=1e-13, max_iter=sweeps)
    k = min(len(r.mar_errs), len(o.mar_errs))
    assert abs(r.niter - o.niter) <= 1
    np.testing.assert_allclose(r.mar_errs[:k], o.mar_errs[:k], rtol=1e-8, atol=1e-13)
    np.testing.assert_allclose(r.obj_vals[:k], o.obj_vals[:k], rtol=0, atol=1e-12)
    np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=1e-11)
    np.testing.assert_allclose(r.plan, o.plan, rtol=0, atol=1e-9 * o.plan.max())


def test_scaled_sweeps_restart_from_a_dual():
    # a start far from the solution: the first launch's base duals do not last
    M, a, b = erot_points(300, 260, seed=4, dtype=np.float64)
    reg = 0.002
    x0 = np.random.default_rng(1).uniform(-0.2, 0.2, 300 + 260 - 1)
    r = regot.sinkhorn_bcd(M, a, b, reg, tol=1e-13, max_iter=40, x0=x0)
    o = O.sinkhorn_bcd(M, a, b, reg, tol=1e-13, max_iter=40, x0=x0)
    assert r.niter == o.niter == 40
    np.testing.assert_allclose(r.mar_errs, o.mar_errs, rtol=1e-8, atol=1e-13)
    np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=1e-11)
