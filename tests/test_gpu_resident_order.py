"""The resident kernels' records and results do not depend on which warp or
block is first: the same bits from run to run, and the oracle's values, at
shapes whose products need no barrier of the block of their own (one cluster
of 16 blocks, wide matrices) and at shapes with a block on every SM."""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")


@pytest.mark.parametrize("n,m", [(80, 700), (15, 4000), (60, 1024), (9, 513)])
def test_bcd_records_in_one_cluster(n, m):
    # errors of z = (alpha + beta - M) / reg as in test_gpu_bcd_scaled.py
    M, a, b = erot_points(n, m, seed=n, dtype=np.float64)
    o = O.sinkhorn_bcd(M, a, b, 0.05, tol=1e-13, max_iter=40)
    P = regot.Problem(M, a, b, precision="fp64")
    first = None
    for _ in range(10):
        r = P.sinkhorn_bcd(0.05, tol=1e-13, max_iter=40)
        k = min(len(r.obj_vals), len(o.obj_vals))
        np.testing.assert_allclose(r.obj_vals[:k], o.obj_vals[:k], rtol=0, atol=1e-12)
        first = r if first is None else first
        assert np.array_equal(r.obj_vals, first.obj_vals)
        assert np.array_equal(r.dual, first.dual)
    P.close()


@pytest.mark.parametrize("n,m", [(40, 30), (90, 700), (300, 260), (1000, 803)])
def test_newton_is_the_same_from_run_to_run(n, m):
    M, a, b = erot_points(n, m, seed=m, dtype=np.float64)
    P = regot.Problem(M, a, b, precision="fp64")
    r = P.sinkhorn_newton(0.02, tol=1e-9, max_iter=50)
    for _ in range(10):
        q = P.sinkhorn_newton(0.02, tol=1e-9, max_iter=50)
        assert np.array_equal(q.obj_vals, r.obj_vals) and np.array_equal(q.dual, r.dual)
    P.close()
