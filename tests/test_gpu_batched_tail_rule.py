"""The batched tail on both sides of its rule (clusters for up to ten problems
of at most sixteen blocks, teams of CTAs beyond, several launches of a team) gives
the bits of the per-sweep kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")


@pytest.mark.parametrize("count,largest", [(7, 512), (10, 512), (10, 513), (11, 300)])
def test_same_bits_as_the_sweep_kernels(count, largest):
    from regot import _lib

    lib = _lib.load()
    rng = np.random.default_rng(count)
    xs, ys, aa, bb = [], [], [], []
    for k in range(count):
        n, m, d = (largest if k == 0 else 40 + 29 * k), 330 - 28 * k, (2, 3, 8, 16)[k % 4]
        xs.append(rng.standard_normal((n, d), dtype=np.float32))
        ys.append(rng.standard_normal((m, d), dtype=np.float32) + np.float32(0.3))
        aa.append(np.full(n, 1.0 / n))
        bb.append(np.full(m, 1.0 / m))
    scale = [1.0 / x.shape[1] for x in xs]
    runs = []
    variant = lib.regot_force_batch_variant(0)  # the arithmetic of the tail
    try:
        for tail in (64, 0):
            old = lib.regot_set_batch_tail(tail)
            try:
                runs.append(regot.sinkhorn_bcd_batched(xs, ys, aa, bb, 0.03, tol=1e-6, max_iter=5000,
                                                       cost_scale=scale, grad=True))
            finally:
                lib.regot_set_batch_tail(old)
    finally:
        lib.regot_force_batch_variant(variant)
    t, s = runs
    assert t.niter.max() > 2 * 64  # more than one launch of a team
    np.testing.assert_array_equal(t.niter, s.niter)
    np.testing.assert_array_equal(t.mar_errs, s.mar_errs)
    np.testing.assert_array_equal(t.costs, s.costs)
    for u, v in zip(t.duals + t.grad_x + t.grad_y, s.duals + s.grad_x + s.grad_y):
        np.testing.assert_array_equal(u, v)
