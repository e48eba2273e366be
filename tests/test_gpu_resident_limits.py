"""Sizes at which a resident kernel's shared memory does not fit fall back to
the captured steps, in the same results."""
import numpy as np
import pytest

from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")


@pytest.mark.parametrize("n", [290000, 300000, 310000])
def test_mixed_newton_systems_at_the_edge_of_shared_memory(n):
    # On 152 SMs the mixed CG's vectors take 228864, 231424 and 233984 bytes a
    # block here: over what is left beside the kernel's static shared memory.
    m, reg = 4, 0.5
    M, a, b = erot_points(n, m, seed=3)
    P = regot.Problem(M, a, b, precision="mixed")
    gamma = np.zeros(n + m - 1)
    rhs = np.random.default_rng(1).standard_normal(n + m - 1)
    x, _ = P.erot_hess_solve(reg, gamma, rhs, tol=1e-8)
    T = np.exp(-M.astype(np.float64) / reg)
    xa, xb = x[:n], np.r_[x[n:], 0.0]
    Hx = np.r_[T.sum(1) * xa + T @ xb, (T.sum(0) * xb + T.T @ xa)[:-1]] / reg
    absH = np.r_[T.sum(1) * abs(xa) + T @ abs(xb), (T.sum(0) * abs(xb) + T.T @ abs(xa))[:-1]] / reg
    # the residual's tolerance and the FP32 plan entries (a few 2^-24 relative)
    assert np.linalg.norm(Hx - rhs) <= 1e-7 * np.linalg.norm(rhs) + 1e-6 * np.linalg.norm(absH)
    r = P.sinkhorn_newton(reg, tol=1e-5, max_iter=30)
    assert r.mar_errs[-1] < 1e-5
    P.close()
