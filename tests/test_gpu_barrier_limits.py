"""The resident kernels' barriers have a limit, and a solve that ran into it ends
with REGOT_ERR_TIMEOUT and leaves its context usable.

The limit is lowered to 0 (regot_set_wait_limit), so that every block leaves at
its first barrier: nothing hangs, and what the blocks had still to write stays
unwritten.
"""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")
from regot import _lib  # noqa: E402

N, M = 300, 260  # a block on every SM, not one cluster


@pytest.fixture
def restore():
    """No waiting, until the test calls this or ends."""
    lib = _lib.load()
    old = lib.regot_set_wait_limit(0)
    yield lambda: lib.regot_set_wait_limit(old)
    lib.regot_set_wait_limit(old)


@pytest.mark.parametrize("solver", ["sinkhorn_bcd", "sinkhorn_newton", "sinkhorn_ssns",
                                    "sinkhorn_sparse_newton", "sinkhorn_splr"])
def test_a_solve_reports_its_barrier(solver, restore):
    C, a, b = erot_points(N, M, seed=4, dtype=np.float64)
    P = regot.Problem(C, a, b, precision="fp64")
    with pytest.raises(RuntimeError, match="blocks gave up"):
        getattr(P, solver)(0.05, tol=1e-8, max_iter=30)
    restore()
    # as if nothing had happened before: the solve of a new problem, bit for bit
    r = getattr(P, solver)(0.05, tol=1e-8, max_iter=30)
    Q = regot.Problem(C, a, b, precision="fp64")
    q = getattr(Q, solver)(0.05, tol=1e-8, max_iter=30)
    assert np.array_equal(r.obj_vals, q.obj_vals) and np.array_equal(r.dual, q.dual)
    # and the oracle's first step, along a direction solved to 1e-8 relative
    # (gradients and steps of the size 1)
    o = getattr(O, solver)(C, a, b, 0.05, tol=1e-8, max_iter=3)
    np.testing.assert_allclose(r.obj_vals[:2], o.obj_vals[:2], rtol=0, atol=1e-6)
    P.close()
    Q.close()


def test_a_hessian_solve_reports_its_barrier(restore):
    C, a, b = erot_points(N, M, seed=4, dtype=np.float64)
    P = regot.Problem(C, a, b, precision="fp64")
    gamma, rhs = np.zeros(N + M - 1), np.ones(N + M - 1)
    with pytest.raises(RuntimeError, match="blocks gave up"):
        P.erot_hess_solve(0.05, gamma, rhs)
    restore()
    x, _ = P.erot_hess_solve(0.05, gamma, rhs, tol=1e-10)
    assert np.linalg.norm(P.erot_hvp(0.05, gamma, x) - rhs) <= 1e-8 * np.linalg.norm(rhs)
    P.close()


def test_a_batch_reports_its_teams_barrier(restore):
    lib = _lib.load()
    rng = np.random.default_rng(0)
    xs = [rng.standard_normal((200 + 40 * k, 3)) for k in range(6)]
    ys = [rng.standard_normal((700 - 50 * k, 3)) for k in range(6)]
    aa = [np.full(len(x), 1.0 / len(x)) for x in xs]
    bb = [np.full(len(y), 1.0 / len(y)) for y in ys]
    variant = lib.regot_force_batch_variant(0)
    try:
        with pytest.raises(RuntimeError, match="gave up"):
            regot.sinkhorn_bcd_batched(xs, ys, aa, bb, 0.5, tol=1e-6, max_iter=2000)
        restore()
        r = regot.sinkhorn_bcd_batched(xs, ys, aa, bb, 0.5, tol=1e-6, max_iter=2000)
    finally:
        lib.regot_force_batch_variant(variant)
    assert np.all(r.mar_errs < 1e-6)
