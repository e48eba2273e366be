"""The FP64 dense passes around the edges of their tiles (16 x 256 up to 2^24
entries, 64 x 256 beyond): row sums, column sums and totals of one pass against
NumPy."""
import numpy as np
import pytest

from problems import erot_points, qrot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")

SHAPES = [(1, 1), (15, 255), (16, 256), (17, 257), (33, 513), (1, 700), (700, 1), (4096, 4096),
          (4097, 4096)]


@pytest.mark.parametrize("n,m", SHAPES)
def test_erot_sums(n, m):
    M, a, b = erot_points(max(n, 2), max(m, 2), seed=n + m, dtype=np.float64)
    M, a, b = np.ascontiguousarray(M[:n, :m]), a[:n] / a[:n].sum(), b[:m] / b[:m].sum()
    rng = np.random.default_rng(5)
    gamma = np.concatenate([0.1 * rng.standard_normal(n + m - 1)])
    reg = 0.1
    T = np.exp((gamma[:n, None] + np.append(gamma[n:], 0.0)[None, :] - M) / reg)
    P = regot.Problem(M, a, b, precision="fp64")
    f, g = P.erot_dual_obj_grad(reg, gamma)
    P.close()
    want = np.concatenate([T.sum(1) - a, (T.sum(0) - b)[:-1]])
    # sums of up to 4097 terms: within 4097 ulp of the largest sum, far less in trees
    np.testing.assert_allclose(g, want, rtol=0, atol=1e-12 * max(T.sum(1).max(), T.sum(0).max()))
    np.testing.assert_allclose(f, reg * T.sum() - a @ gamma[:n] - b[:-1] @ gamma[n:], rtol=1e-12)


@pytest.mark.parametrize("n,m", SHAPES)
def test_qrot_sums(n, m):
    M, a, b = qrot_points(max(n, 2), max(m, 2), seed=n + m, dtype=np.float64)
    M, a, b = np.ascontiguousarray(M[:n, :m]), a[:n] / a[:n].sum(), b[:m] / b[:m].sum()
    rng = np.random.default_rng(6)
    gamma = 0.3 + 0.2 * rng.standard_normal(n + m)
    reg = 0.1
    D = np.maximum(gamma[:n, None] + gamma[n:][None, :] - M, 0.0)
    P = regot.Problem(M, a, b, precision="fp64")
    f, g = P.qrot_dual_obj_grad(reg, gamma)
    P.close()
    want = np.concatenate([D.sum(1) - reg * a, D.sum(0) - reg * b])
    np.testing.assert_allclose(g, want, rtol=0, atol=1e-12 * max(D.sum(1).max(), D.sum(0).max()))
    want_f = 0.5 * (D * D).sum() - reg * (a @ gamma[:n] + b @ gamma[n:])
    np.testing.assert_allclose(f, want_f, rtol=1e-12, atol=1e-12)
