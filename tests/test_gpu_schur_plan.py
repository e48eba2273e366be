"""FP64 SSNS on the stored plan and the one-launch Schur CG
(csrc/schur_plan.cuh) against the FP64 oracle, at the edges of the launch
shapes (one cluster up to 65536 entries, a block an SM beyond; fewer rows or
columns than blocks or warps), with both linear solvers."""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")

SHAPES = [(5, 1), (1, 5), (2, 3), (16, 65), (31, 33), (3, 900), (900, 3), (256, 256), (257, 256),
          (151, 701), (700, 95)]


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("n,m", SHAPES)
def test_ssns_reaches_the_oracle_solution(n, m, method):
    # both stop at a marginal error below 1e-9; near the optimum the duals
    # differ by that over the smallest curvature, plan entries by less
    M, a, b = erot_points(n, m, seed=n + m, dtype=np.float64)
    reg = 0.05
    r = regot.sinkhorn_ssns(M, a, b, reg, tol=1e-9, max_iter=400, method=method)
    o = O.sinkhorn_ssns(M, a, b, reg, tol=1e-9, max_iter=400, method=method)
    assert (r.mar_errs[-1] < 1e-9) == (o.mar_errs[-1] < 1e-9)
    assert len(r.densities) == len(r.mar_errs) == r.niter + 1
    np.testing.assert_allclose(r.obj_vals[0], o.obj_vals[0], rtol=0, atol=1e-12)
    np.testing.assert_allclose(r.mar_errs[0], o.mar_errs[0], rtol=1e-10, atol=1e-14)
    if m > 1:  # without a beta block the solver reports 1 and the oracle 1 / n
        np.testing.assert_allclose(r.densities[0], o.densities[0], rtol=1e-12)
    np.testing.assert_allclose(r.obj_vals[-1], o.obj_vals[-1], rtol=0, atol=1e-9)
    np.testing.assert_allclose(r.plan, o.plan, rtol=0, atol=1e-6 * o.plan.max())


@pytest.mark.parametrize("n,m", [(64, 48), (300, 260)])
def test_first_ssns_step_is_the_oracle_step(n, m):
    # one direction, line selection and gradient from the same start: the
    # Schur CG of method 1 (1e-10) against the oracle's factorisation
    M, a, b = erot_points(n, m, seed=7, dtype=np.float64)
    r = regot.sinkhorn_ssns(M, a, b, 0.05, tol=1e-12, max_iter=1)
    o = O.sinkhorn_ssns(M, a, b, 0.05, tol=1e-12, max_iter=1)
    np.testing.assert_allclose(r.mar_errs, o.mar_errs, rtol=1e-7)
    np.testing.assert_allclose(r.obj_vals, o.obj_vals, rtol=0, atol=1e-10)
    np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=1e-8)
