"""The batched tail in teams of CTAs (one cooperative launch): uneven problems,
down to a single point and beyond sixteen blocks of rows or columns, give the
bits of the per-sweep kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")

BATCHES = {
    "one-large": [(700, 530, 3)],
    "edges": [(1, 1, 2), (1, 600, 3), (600, 1, 3), (31, 33, 8), (32, 32, 16), (513, 512, 2)],
    "many": [(20 + 11 * k, 500 - 7 * k, (2, 3, 4, 6, 8, 12, 16)[k % 7]) for k in range(60)],
}


@pytest.mark.parametrize("batch", list(BATCHES))
def test_same_bits_as_the_sweep_kernels(batch):
    from regot import _lib

    rng = np.random.default_rng(3)
    xs, ys, as_, bs, scale = [], [], [], [], []
    for n, m, d in BATCHES[batch]:
        xs.append(rng.standard_normal((n, d), dtype=np.float32))
        ys.append(rng.standard_normal((m, d), dtype=np.float32) + np.float32(0.3))
        a, b = rng.uniform(0.5, 1.5, n), rng.uniform(0.5, 1.5, m)
        as_.append(a / a.sum())
        bs.append(b / b.sum())
        scale.append(1.0 / d)
    lib = _lib.load()
    # the tail has the arithmetic of the CUDA-core half-sweeps
    variant = lib.regot_force_batch_variant(0)
    runs = []
    for tail in (64, 0):
        old = lib.regot_set_batch_tail(tail)
        try:
            runs.append(regot.sinkhorn_bcd_batched(xs, ys, as_, bs, 0.05, tol=1e-6, max_iter=3000,
                                                   cost_scale=scale, grad=True))
        finally:
            lib.regot_set_batch_tail(old)
            if tail == 0 or len(runs) < 1:
                lib.regot_force_batch_variant(variant)
    t, s = runs
    np.testing.assert_array_equal(t.niter, s.niter)
    np.testing.assert_array_equal(t.mar_errs, s.mar_errs)
    for u, v in zip(t.duals, s.duals):
        np.testing.assert_array_equal(u, v)
    np.testing.assert_array_equal(t.costs, s.costs)
