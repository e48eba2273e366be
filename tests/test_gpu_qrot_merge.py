"""The merge of qrot_lbfgs_dual's line-search trials and the primal value's
merges at the edges of their blocks (64 items a block, 32 rows or columns, 64
partials a piece: 4096 rows of FP32, 1024 of FP64), against the FP64 oracle."""
import numpy as np
import pytest

import regot_oracle as O
from problems import qrot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")

SHAPES = [(2, 2), (5, 3), (31, 33), (33, 31), (64, 64), (65, 63), (40, 600), (1024, 17),
          (1025, 17), (1100, 20), (4200, 30)]
ITERS = 5


@pytest.mark.parametrize("n,m", SHAPES)
def test_fp64_first_iterations(n, m):
    M, a, b = qrot_points(n, m, seed=n + m, dtype=np.float64)
    r = regot.qrot_lbfgs_dual(M, a, b, 0.1, tol=1e-14, max_iter=ITERS, precision="fp64")
    o = O.qrot_lbfgs_dual(M, a, b, 0.1, tol=1e-14, max_iter=ITERS)
    # rounding differences of some 1e-15 double in an iteration; sums of up
    # to 4230 terms
    assert r.niter == o.niter
    np.testing.assert_allclose(r.obj_vals, o.obj_vals, rtol=1e-10, atol=1e-12)
    np.testing.assert_allclose(r.mar_errs, o.mar_errs, rtol=1e-8, atol=1e-12)
    np.testing.assert_allclose(r.prim_vals, o.prim_vals, rtol=1e-8, atol=1e-12)
    np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=1e-10 * max(1, np.abs(o.dual).max()))


@pytest.mark.parametrize("n,m", SHAPES)
def test_mixed_first_iterations(n, m):
    M, a, b = qrot_points(n, m, seed=n + m, dtype=np.float64)
    Mq = M.astype(np.float32).astype(np.float64)
    r = regot.qrot_lbfgs_dual(M, a, b, 0.1, tol=1e-14, max_iter=ITERS, precision="mixed")
    o = O.qrot_lbfgs_dual(Mq, a, b, 0.1, tol=1e-14, max_iter=ITERS)
    assert r.niter == o.niter
    # FP32 sums: 1e-7 relative, doubling an iteration, with a margin of 30
    np.testing.assert_allclose(r.obj_vals, o.obj_vals, rtol=1e-4, atol=1e-8)
    np.testing.assert_allclose(r.prim_vals, o.prim_vals, rtol=1e-4, atol=1e-8)
    np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=1e-4 * max(1, np.abs(o.dual).max()))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("solver", ["qrot_lbfgs_dual", "qrot_assn"])
def test_primal_value_is_that_of_the_dual(solver, precision):
    # two passes from the gradient's row sums against the three of
    # qrot_primal_val at the same duals
    M, a, b = qrot_points(300, 210, seed=4, dtype=np.float64)
    P = regot.Problem(M, a, b, precision=precision)
    r = getattr(P, solver)(0.1, tol=1e-14, max_iter=12, plan=False)
    want = P.qrot_primal_val(0.1, r.dual)
    P.close()
    np.testing.assert_allclose(r.prim_vals[-1], want, rtol=1e-11 if precision == "fp64" else 2e-6)
