"""Every device allocation of a solve made to fail in turn (regot_fail_allocation).

A solve either ends in RuntimeError or, where what could not be had is a second
matrix or an engine beside the first, falls back to the passes and gives the
oracle's result. Either way the problem then solves as if nothing had happened.
"""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points, qrot_points, readme_example

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")
from regot import _lib  # noqa: E402

DEAD = np.r_[np.full(100, -40.0), np.zeros(79)]  # row sums that all underflow at reg 0.05


def _scan(make, solve, check):
    """Outcomes of the solves with allocation 1, 2, ... failing, up to the first
    that reaches none: True where the solve succeeded all the same."""
    lib = _lib.load()
    outcomes = []
    for k in range(1, 400):
        P = make()
        lib.regot_fail_allocation(k)
        try:
            r = solve(P)
            ok = True
        except RuntimeError as e:
            assert "regot_fail_allocation" in str(e)
            ok = False
        finally:
            left = lib.regot_fail_allocation(0)
        if ok:
            check(r)
        else:
            check(solve(P))
        P.close()
        if left:
            return outcomes
        outcomes.append(ok)
    raise AssertionError("no solve without a failing allocation")


# problem, solver, its options, how far results may be off, fallbacks at least
ENTROPIC = [
    # a matrix (K or T) and its buffers; of SSNS also those of the Schur CG
    ("points", "fp64", "sinkhorn_bcd", dict(reg=0.05, tol=1e-9, max_iter=400), 1e-8, 3),
    ("readme", "fp64", "sinkhorn_bcd", dict(reg=0.05, tol=1e-9, max_iter=3000, x0=DEAD), 1e-7, 3),
    ("points", "fp64", "sinkhorn_newton", dict(reg=0.05, tol=1e-9, max_iter=50), 1e-8, 4),
    ("points", "mixed", "sinkhorn_newton", dict(reg=0.05, tol=1e-6, max_iter=50), 1e-4, 2),
    ("points", "fp64", "sinkhorn_ssns", dict(reg=0.05, tol=1e-9, max_iter=200), 1e-7, 5),
    ("points", "mixed", "sinkhorn_bcd", dict(reg=0.05, tol=1e-6, max_iter=400), 1e-4, 0),
]


@pytest.mark.parametrize("problem,precision,solver,options,atol,fallbacks", ENTROPIC)
def test_entropic_solves(problem, precision, solver, options, atol, fallbacks):
    # Duals of a solve to marginal error tol: the dual Hessian's entries are
    # marginals over reg (1 / (300 * 0.05) here), so a gradient of tol leaves about
    # 15 tol in a dual; the bounds have a factor of five and more on top, the
    # README example's (marginals down to 1e-3 of the mean) a hundred.
    if problem == "points":
        M, a, b = erot_points(300, 260, seed=4)
    else:
        M, a, b = readme_example(100, 80)
    M = M.astype(np.float64)
    o = getattr(O, solver)(M, a, b, **options)
    assert o.mar_errs[-1] < options["tol"]

    def check(r):
        assert r.mar_errs[-1] < options["tol"]
        np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=atol)

    outcomes = _scan(lambda: regot.Problem(M, a, b, precision=precision),
                     lambda P: getattr(P, solver)(**options), check)
    assert sum(outcomes) >= fallbacks and outcomes.count(False) >= 5


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("solver", ["qrot_lbfgs_dual", "qrot_assn", "qrot_grssn"])
def test_quadratic_solves(solver, precision):
    # the primal values' second engine is left out where it has no room: the same
    # kernels then run one after another, so every value has the same bits
    M, a, b = qrot_points(150, 130, seed=2)
    P = regot.Problem(M, a, b, precision=precision)
    want = getattr(P, solver)(0.1, tol=1e-6, max_iter=8)
    P.close()
    assert len(want.prim_vals) >= 4

    def check(r):
        assert np.array_equal(r.prim_vals, want.prim_vals)
        assert np.array_equal(r.obj_vals, want.obj_vals)
        assert np.array_equal(r.dual, want.dual)

    outcomes = _scan(lambda: regot.Problem(M, a, b, precision=precision),
                     lambda P: getattr(P, solver)(0.1, tol=1e-6, max_iter=8), check)
    assert sum(outcomes) >= 5 and outcomes.count(False) >= 5
