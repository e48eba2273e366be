"""The QROT Schur CG on index lists at the edges of its slices: one to eight rows
or columns a thread (256 threads on 16 blocks), blocks without any, a row or a
column alone, against the bitmask path and the FP64 oracle."""
import numpy as np
import pytest

import regot_oracle as O
from problems import qrot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")

# (with a single row the initial value is the solution: no step to compare)
SHAPES = [(40, 1), (3, 70), (33, 31), (4096, 40), (4200, 40), (40, 4200), (9000, 30),
          (17000, 20)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n,m", SHAPES)
def test_first_newton_steps(n, m, precision):
    from regot import _lib

    lib = _lib.load()
    M, a, b = qrot_points(n, m, seed=n + m, dtype=np.float64)
    Mq = M.astype(np.float32).astype(np.float64) if precision == "mixed" else M
    runs = {}
    for mode in (1, 2):  # bitmask, index lists
        old = lib.regot_force_qrot_cg_path(mode)
        try:
            runs[mode] = regot.qrot_assn(M, a, b, 0.1, tol=1e-12, max_iter=3, precision=precision)
        finally:
            lib.regot_force_qrot_cg_path(old)
    o = O.qrot_assn(Mq, a, b, 0.1, tol=1e-12, max_iter=3)
    # CG to 1e-8 on both paths; FP32 passes to 1e-7, magnified by the steps
    rt = 1e-5 if precision == "fp64" else 1e-2
    assert runs[2].niter == runs[1].niter
    np.testing.assert_allclose(runs[2].mar_errs, runs[1].mar_errs, rtol=rt, atol=1e-6)
    np.testing.assert_allclose(runs[2].mar_errs, o.mar_errs, rtol=rt, atol=1e-6)
    np.testing.assert_allclose(runs[2].obj_vals, o.obj_vals, rtol=rt, atol=1e-6)
