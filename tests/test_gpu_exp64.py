"""The FP64 plan entries exp((alpha_i + beta_j - M_ij) / reg) (csrc/exp64.cuh)
against NumPy's extended-precision exponential, over the whole range of
exponents and at its ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")


def _plan(Z):
    """exp(Z) through erot_plan: reg = 1, gamma = 0, M = -Z (all exact)."""
    n, m = Z.shape
    P = regot.Problem(-Z, np.full(n, 1.0 / n), np.full(m, 1.0 / m), precision="fp64")
    T = np.array(P.erot_plan(1.0, np.zeros(n + m - 1)))
    P.close()
    return T


@pytest.mark.parametrize("lo,hi", [(-1.0, 1.0), (-40.0, 0.0), (-700.0, 700.0), (-1e-8, 1e-8)])
@pytest.mark.parametrize("shape", [(64, 65), (200, 300)])
def test_within_an_ulp(lo, hi, shape):
    Z = np.random.default_rng(3).uniform(lo, hi, shape)
    Z[0, :2] = lo, hi
    T = _plan(Z)
    want = np.exp(Z.astype(np.longdouble))
    # one unit in the last place, of a significand between 1 and 2: 2^-52 at most
    assert np.max(np.abs(T / want - 1)) <= 2.0 ** -52


def test_ends_of_the_range():
    z = np.array([[0.0, -707.9, -708.0, -708.4, -720.0, -744.9, -745.2, -746.1, -800.0, -1e5, -1e300],
                  [707.9, 708.0, 709.7, 1e-300, -1e-300, -1.0, 1.0, -745.9, -747.0, -1e10, -709.0]])
    T = _plan(z)
    with np.errstate(under="ignore"):
        want = np.exp(z)
    # the smallest results are denormal: one unit there is 2^-1074
    np.testing.assert_allclose(T, want, rtol=2.0 ** -52, atol=2.0 ** -1074)
    assert np.all(T[z < -746] == 0.0)


def test_line_search_sums_on_the_plan():
    """The Armijo sums of the FP64 Newton solver use phi(x) = e^x - 1 - x from a
    table; a solve whose steps span tiny and large arguments takes the oracle's
    path (accepted steps show in the objectives)."""
    import regot_oracle as O
    from problems import erot_points

    M, a, b = erot_points(300, 260, seed=9, dtype=np.float64)
    r = regot.sinkhorn_newton(M, a, b, 0.01, tol=1e-8, max_iter=50)
    o = O.sinkhorn_newton(M, a, b, 0.01, tol=1e-8, max_iter=50)
    k = sum(1 for v in o.mar_errs if v > 1e-6)  # before the rounding floor
    assert r.mar_errs[-1] < 1e-8
    np.testing.assert_allclose(r.obj_vals[:k], o.obj_vals[:k], rtol=0, atol=1e-9)
