"""FP64 sinkhorn_bcd where the scalings of its stored plan grow beyond what the
plan's entries can carry.

The plan K is formed at the start's duals; an entry below the range of a double is
lost. A row whose sum is 2^-866 gets the scaling 2^865, and then a column whose
largest contribution was one of that row's lost entries must not be summed from
the rest.
"""
import numpy as np
import pytest

import regot_oracle as O

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")


def _lost_entry(n, m, row_cost, lost, other):
    # row 0 costs row_cost in every column but the last two, where it costs `lost`
    # (exp(-lost) underflows); the other rows cost 0, and `other` in those two
    M = np.zeros((n, m))
    M[1:, m - 2:] = other
    M[0] = row_cost
    M[0, m - 2:] = lost
    return M, np.full(n, 1.0 / n), np.full(m, 1.0 / m)


@pytest.mark.parametrize("n,m", [(2, 3), (40, 30), (300, 260)])
@pytest.mark.parametrize("row_cost,lost,other", [(600.0, 800.0, 500.0), (340.0, 760.0, 600.0),
                                                 (330.0, 700.0, 300.0)])
@pytest.mark.parametrize("sweeps", [1, 2, 3])
def test_a_column_of_lost_entries_follows_the_oracle(n, m, row_cost, lost, other, sweeps):
    # From the duals 0 at reg = 1 the arguments are the costs, below 2^10: the
    # exponentials' arguments round by 2^-43, T by that relatively, a sum and its
    # logarithm by about as much; three sweeps of them stay below 1e-11.
    M, a, b = _lost_entry(n, m, row_cost, lost, other)
    x0 = np.zeros(n + m - 1)
    o = O.sinkhorn_bcd(M, a, b, 1.0, tol=1e-13, max_iter=sweeps, x0=x0)
    r = regot.sinkhorn_bcd(M, a, b, 1.0, tol=1e-13, max_iter=sweeps, x0=x0)
    assert r.niter == o.niter
    np.testing.assert_allclose(r.dual, o.dual, rtol=1e-12, atol=1e-10)
    np.testing.assert_allclose(r.mar_errs, o.mar_errs, rtol=1e-9, atol=1e-13)
    np.testing.assert_allclose(r.plan, o.plan, rtol=0, atol=1e-10)
