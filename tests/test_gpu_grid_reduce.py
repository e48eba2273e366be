"""Grid-wide sums over one block to more than 256 (warp_grid_reduce), at the
edges of its rounds of loads: the marginal errors and objectives of mixed BCD
(blocks of 32 rows or columns) and the primal values of QROT against the
oracle."""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points, qrot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")

SIZES = [1, 31, 1024, 1025, 2048, 2049, 8192, 8193]  # 1, 1, 32, 33, 64, 65, 256, 257 blocks


@pytest.mark.parametrize("long", SIZES)
@pytest.mark.parametrize("tall", [True, False])
def test_bcd_records(long, tall):
    n, m = (long, 9) if tall else (9, long)
    if m == 1:
        pytest.skip("a single column leaves nothing to iterate")
    M, a, b = erot_points(n, m, seed=long)
    reg = 0.1
    r = regot.sinkhorn_bcd(M, a, b, reg, tol=1e-13, max_iter=4, precision="mixed")
    o = O.sinkhorn_bcd(M.astype(np.float64), a, b, reg, tol=1e-13, max_iter=4)
    k = min(len(r.mar_errs), len(o.mar_errs))
    # plan entries in FP32 at arguments up to 1 / reg = 10: 1e-6 relative to the
    # marginals, whose norm is below 1; objectives of the size 1
    np.testing.assert_allclose(r.mar_errs[:k], o.mar_errs[:k], rtol=0, atol=2e-6)
    np.testing.assert_allclose(r.obj_vals[:k], o.obj_vals[:k], rtol=0, atol=2e-6)


@pytest.mark.parametrize("long", [31, 1024, 1025, 2048, 2049, 8192, 8193])
def test_qrot_primal_values(long):
    M, a, b = qrot_points(long, 9, seed=long, dtype=np.float64)
    gamma = np.random.default_rng(3).uniform(0.0, 0.5, long + 9)
    P = regot.Problem(M, a, b, precision="fp64")
    got, want = P.qrot_primal_val(0.1, gamma), O.qrot_primal_val(M, a, b, 0.1, gamma)
    # sums of 10^5 FP64 terms of one sign
    assert abs(got - want) <= 1e-11 * max(1.0, abs(want))
    P.close()
