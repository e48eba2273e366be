"""FP64 Newton and Hessian solves on the stored plan (csrc/newton_plan.cuh) and
the FP64 column sums of optimal_beta against the FP64 oracle, at the edges of
their launch shapes."""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")

SHAPES = [(1, 5), (5, 1), (2, 2), (16, 65), (31, 33), (3, 900), (900, 3), (256, 256), (257, 256),
          (151, 701), (153, 1030), (700, 95)]


@pytest.mark.parametrize("n,m", SHAPES)
def test_newton_on_the_plan_follows_the_oracle(n, m):
    # the directions agree to the CG tolerance (1e-10), the duals at the
    # solution to that times their size and the last step's; the number of
    # iterations need not (near the solution the two line searches see
    # objective changes at the rounding of their different forms)
    reg = 0.05
    M, a, b = erot_points(n, m, seed=n + m, dtype=np.float64)
    r = regot.sinkhorn_newton(M, a, b, reg, tol=1e-9, max_iter=50)
    o = O.sinkhorn_newton(M, a, b, reg, tol=1e-9, max_iter=50)
    assert r.mar_errs[-1] < 1e-9 and len(r.mar_errs) == len(r.obj_vals) == r.niter + 1
    np.testing.assert_allclose(r.obj_vals[-1], o.obj_vals[-1], rtol=0, atol=1e-9)
    np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=1e-9)
    np.testing.assert_allclose(r.plan, o.plan, rtol=0, atol=1e-7 * o.plan.max())
    r1 = regot.sinkhorn_newton(M, a, b, reg, tol=1e-9, max_iter=1)
    o1 = O.sinkhorn_newton(M, a, b, reg, tol=1e-9, max_iter=1)
    assert r1.niter == o1.niter
    np.testing.assert_allclose(r1.mar_errs, o1.mar_errs, rtol=1e-7, atol=1e-12)


@pytest.mark.parametrize("n,m", SHAPES)
def test_hessian_solve_on_the_plan(n, m):
    # x solves H x = rhs to the CG tolerance: the residual by the oracle's
    # own Hessian product
    reg = 0.05
    M, a, b = erot_points(n, m, seed=n + m, dtype=np.float64)
    gamma = O.sinkhorn_bcd(M, a, b, reg, tol=1e-6, max_iter=500, plan=False).dual
    rhs = np.random.default_rng(0).standard_normal(n + m - 1)
    P = regot.Problem(M, a, b)
    x, steps = P.erot_hess_solve(reg, gamma, rhs, tol=1e-11)
    assert steps > 0
    res = O.erot_hvp(M, a, b, reg, gamma, x) - rhs
    assert np.linalg.norm(res) < 1e-9 * np.linalg.norm(rhs)
    P.close()


@pytest.mark.parametrize("n,m", [(1, 1), (64, 32), (65, 33), (130, 200), (1000, 7)])
def test_optimal_beta_fp64_shapes(n, m):
    M, a, b = erot_points(n, m, seed=3, dtype=np.float64)
    alpha = np.random.default_rng(1).standard_normal(n) * 0.1
    P = regot.Problem(M, a, b)
    np.testing.assert_allclose(P.erot_optimal_beta(0.02, alpha),
                               O.erot_optimal_beta(M, b, 0.02, alpha), rtol=0, atol=1e-13)
    P.close()


SHAPES32 = [(1, 5), (5, 1), (63, 511), (64, 512), (65, 513), (129, 1030), (300, 260), (2100, 1000),
            (40, 4200), (4200, 40)]


@pytest.mark.parametrize("n,m", SHAPES32)
def test_mixed_hessian_solve_on_the_plan(n, m):
    # T carries a few 1e-7 relative and the FP32 tile sums some 1e-7 more, so a
    # product errs by less than 5e-7 of H |x|; the residual that CG updates
    # drifts from the true one by a few products' errors: four of them, and
    # the solve's own tolerance
    reg = 0.05
    M, a, b = erot_points(n, m, seed=n + m, dtype=np.float32)
    Mq = M.astype(np.float64)
    gamma = O.sinkhorn_bcd(Mq, a, b, reg, tol=1e-5, max_iter=200, plan=False).dual
    rhs = np.random.default_rng(0).standard_normal(n + m - 1)
    P = regot.Problem(M, a, b, precision="mixed")
    x, steps = P.erot_hess_solve(reg, gamma, rhs, tol=1e-7)
    assert steps > 0
    res = O.erot_hvp(Mq, a, b, reg, gamma, x) - rhs
    size = O.erot_hvp(Mq, a, b, reg, gamma, np.abs(x))
    assert np.linalg.norm(res) < 2e-6 * np.linalg.norm(size) + 1e-7 * np.linalg.norm(rhs)
    P.close()


@pytest.mark.parametrize("n,m", [(65, 513), (700, 1100)])
def test_mixed_newton_on_the_plan_agrees_with_fp64(n, m):
    reg = 0.05
    M, a, b = erot_points(n, m, seed=n + m, dtype=np.float32)
    r = regot.sinkhorn_newton(M, a, b, reg, tol=1e-6, max_iter=50, precision="mixed")
    o = regot.sinkhorn_newton(M.astype(np.float64), a, b, reg, tol=1e-6, max_iter=50)
    assert r.mar_errs[-1] < 1e-6
    np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=1e-6)
