"""Shared memory of the resident kernels: sizes at which it does not fit fall back
to the captured steps, and solves of different sizes run beside each other."""
import threading

import numpy as np
import pytest

from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")
from regot import _lib  # noqa: E402

_thread = threading.local()


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


def _solves(solver, precision, sizes, reg, count, errors, results, **kw):
    """`count` solves of each size in turn, in a context of this thread's own."""
    try:
        ctx = _lib.Context(0)
        _thread.ctx = ctx
        for n, m in sizes:
            M, a, b = erot_points(n, m, seed=n, dtype=np.float64)
            P = regot.Problem(M, a, b, precision=precision)
            for _ in range(count):
                results.append((n, getattr(P, solver)(reg, **kw).dual))
            P.close()
    except Exception as e:  # noqa: BLE001 - reported by the test's thread
        errors.append(repr(e))


# sizes whose kernels ask for different amounts of shared memory
@pytest.mark.parametrize("solver,precision,kw", [
    ("sinkhorn_newton", "mixed", dict(tol=1e-5, max_iter=20)),
    ("sinkhorn_newton", "fp64", dict(tol=1e-8, max_iter=20)),
    ("sinkhorn_bcd", "fp64", dict(tol=1e-8, max_iter=60)),
    ("sinkhorn_ssns", "fp64", dict(tol=1e-8, max_iter=200)),
    ("sinkhorn_ssns", "mixed", dict(tol=1e-5, max_iter=200)),
])
def test_two_threads_solve_two_sizes_at_once(solver, precision, kw, monkeypatch):
    monkeypatch.setattr(_lib, "context", lambda device=0: _thread.ctx)
    sizes = [(2000, 2000), (600, 9000), (200, 210)]
    errors, results = [], [[], []]
    threads = [threading.Thread(target=_solves, args=(solver, precision, s, 0.05, 12, errors, r),
                                kwargs=kw)
               for s, r in zip((sizes, sizes[::-1]), results)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert errors == []
    # the other thread's results, whatever ran beside: solves of the same problem,
    # converged to a marginal error of 1e-5 at most (duals of order one)
    for n, _ in sizes:
        duals = [d for r in results for k, d in r if k == n]
        assert len(duals) == 24
        for d in duals[1:]:
            np.testing.assert_allclose(d, duals[0], rtol=0, atol=1e-6)
