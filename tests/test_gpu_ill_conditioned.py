"""Conjugate gradients of many steps on ill-conditioned systems: the Newton systems
of FP64 EROT near the solution at a small regularisation, and the shifted
systems of QROT, whose resident kernels form p'Hp from half of the products
(and, for QROT, carry the rows' products along), leave residuals as small as the
condition allows."""
import numpy as np
import pytest

import regot_oracle as O
from problems import erot_points, qrot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")


# condition 3e3 (one cluster), 4e4 and 6e8 (a block an SM); 110 to 400 steps
@pytest.mark.parametrize("n,m,reg,sweeps", [(60, 50, 0.0005, 100), (600, 500, 0.002, 50),
                                            (600, 500, 0.001, 100)])
def test_newton_systems(n, m, reg, sweeps):
    M, a, b = erot_points(n, m, seed=1, dtype=np.float64)
    g = O.sinkhorn_bcd(M, a, b, reg, tol=0, max_iter=sweeps).dual
    T = np.exp((g[:n, None] + np.r_[g[n:], 0.0] - M) / reg)
    H = np.diag(np.r_[T.sum(1), T.sum(0)[:-1]]) / reg
    H[:n, n:] = T[:, :-1] / reg
    H[n:, :n] = H[:n, n:].T
    w = np.linalg.eigvalsh(H)
    rhs = np.random.default_rng(2).standard_normal(n + m - 1)
    P = regot.Problem(M, a, b, precision="fp64")
    for tol in (1e-8, 1e-12):
        x, steps = P.erot_hess_solve(reg, g, rhs, tol=tol)
        assert steps > 50
        # the steps' tolerance, and the rounding of products with x
        assert np.linalg.norm(H @ x - rhs) <= (tol + 2.3e-16 * w[-1] / w[0]) * np.linalg.norm(rhs)
    P.close()


@pytest.mark.parametrize("n,m", [(60, 50), (300, 260), (1023, 769)])
@pytest.mark.parametrize("shift", [1e-2, 1e-4, 1e-6])
def test_shifted_qrot_systems(n, m, shift, qrot_cg_path):
    M, a, b = qrot_points(n, m, seed=1, dtype=np.float64)
    x0 = O.qrot_grssn(M, a, b, 0.1, tol=1e-12, max_iter=6).dual
    g = O.qrot_dual_obj_grad(M, a, b, 0.1, x0)[1]
    S = (x0[:n, None] + x0[None, n:] - M > 0).astype(float)
    A = np.diag(np.r_[S.sum(1), S.sum(0)] + shift)
    A[:n, n:] = S
    A[n:, :n] = S.T
    d = np.linalg.solve(A, -g)
    r = regot.qrot_grssn(M, a, b, 0.1, tol=0, max_iter=1, x0=x0, shift=shift, precision="fp64")
    # the direction, from the step: a power of 1/2 of the line search
    e = r.dual - x0
    e /= 2.0 ** np.round(np.log2(e @ d / (d @ d)))
    # CG stops at 1e-8 of its right-hand side; the difference of the duals has
    # rounding of 1e-16 over the step (4e-6 at the smallest shift)
    assert np.linalg.norm(A @ e + g) <= 2e-8 * np.linalg.norm(g)
