"""The resident kernels' records and results do not depend on which warp or
block is first: the same bits from run to run, and the oracle's values, at
shapes whose products need no barrier of the block of their own (one cluster
of 16 blocks up to 24576 entries, wide matrices) and at shapes with a block on
every SM."""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")


@pytest.mark.parametrize("n,m", [(35, 700), (6, 4000), (20, 1024), (9, 513), (15, 4000)])
def test_bcd_records(n, m):
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


@pytest.mark.parametrize("n,m", [(40, 30), (30, 700), (128, 192), (193, 128), (300, 260), (1000, 803)])
def test_newton_is_the_same_from_run_to_run(n, m):
    M, a, b = erot_points(n, m, seed=m, dtype=np.float64)
    P = regot.Problem(M, a, b, precision="fp64")
    r = P.sinkhorn_newton(0.02, tol=1e-9, max_iter=50)
    for _ in range(10):
        q = P.sinkhorn_newton(0.02, tol=1e-9, max_iter=50)
        assert np.array_equal(q.obj_vals, r.obj_vals) and np.array_equal(q.dual, r.dual)
    P.close()


@pytest.mark.parametrize("n,m,reg", [(100, 80, 0.05), (33, 2000, 0.02), (3000, 400, 0.01),
                                     (2049, 2049, 0.01)])
def test_first_record_from_a_dual_off_the_split_grid(n, m, reg):
    # Mixed precision from a dual far below its final size: the first row update
    # leaves the grid of the FP32 splits, iterate 0 is handed to the general path
    # unrecorded, and its marginal error keeps the column part, which only a user's
    # dual has. The FP32 sums of the plan entries (FP32 exponentials at arguments
    # up to 1 / reg: a few 1e-6 relative each) bound the difference.
    M, a, b = erot_points(n, m, seed=5)
    x0 = np.full(n + m - 1, 1e-4)
    o = O.sinkhorn_bcd(M.astype(np.float64), a, b, reg, tol=1e-13, max_iter=2, x0=x0)
    T = np.exp((2e-4 - M.astype(np.float64)) / reg)
    T[:, -1] = np.exp((1e-4 - M[:, -1].astype(np.float64)) / reg)
    rows, cols = T.sum(1) - a, (T.sum(0) - b)[:-1]
    want = np.sqrt((rows ** 2).sum() + (cols ** 2).sum())
    np.testing.assert_allclose(o.mar_errs[0], want, rtol=1e-9)
    assert (cols ** 2).sum() > 0.01 * want ** 2  # the part that could go missing
    P = regot.Problem(M, a, b, precision="mixed")
    first = None
    for _ in range(25):
        r = P.sinkhorn_bcd(reg, tol=1e-13, max_iter=2, x0=x0)
        np.testing.assert_allclose(r.mar_errs[0], want, rtol=1e-4)
        first = r if first is None else first
        assert np.array_equal(r.mar_errs, first.mar_errs)
        assert np.array_equal(r.obj_vals, first.obj_vals)
        assert np.array_equal(r.dual, first.dual)
    P.close()


@pytest.mark.parametrize("n,m", [(128, 192), (193, 128), (24576, 1), (1, 24577), (24577, 1)])
def test_the_edge_of_one_cluster(n, m):
    # 24576 entries run in one cluster, more in a block an SM (errors as above)
    M, a, b = erot_points(n, m, seed=7, dtype=np.float64)
    o = O.sinkhorn_bcd(M, a, b, 0.05, tol=1e-13, max_iter=20)
    r = regot.sinkhorn_bcd(M, a, b, 0.05, tol=1e-13, max_iter=20)
    k = min(len(r.obj_vals), len(o.obj_vals))
    assert abs(r.niter - o.niter) <= 1
    np.testing.assert_allclose(r.obj_vals[:k], o.obj_vals[:k], rtol=0, atol=1e-12)
    np.testing.assert_allclose(r.dual, o.dual, rtol=0, atol=1e-11)
