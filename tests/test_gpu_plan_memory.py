"""The stored plan's memory is given back before the plan is written out.

A process of its own, whose memory pool starts empty and keeps what it mapped,
solves once with the plan into plain host memory (which goes through a device
buffer of the plan's size): the pool has then mapped the cost matrix, and one
matrix more, which was the stored plan first and the output afterwards.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("regot")

CODE = """
import sys
sys.path[:0] = %r
import numpy as np, torch
import regot
from regot import _lib
from problems import erot_points

_lib.host_empty = lambda shape, dtype=np.float64: np.empty(shape, dtype)
M, a, b = erot_points(50, 40, seed=1, dtype=np.float64)
for solver in (regot.sinkhorn_bcd, regot.sinkhorn_newton):
    solver(M, a, b, 0.1)
M, a, b = erot_points(5000, 4800, seed=1, dtype=np.float64)
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
r = getattr(regot, %r)(M, a, b, 0.1, tol=1e-6, max_iter=50)
used = before - torch.cuda.mem_get_info()[0]
assert r.plan.shape == M.shape and abs(r.plan.sum() - 1.0) < 1e-5
print("matrices", used / M.nbytes)
"""


@pytest.mark.parametrize("solver", ["sinkhorn_bcd", "sinkhorn_newton"])
def test_one_matrix_beside_the_cost(solver):
    here = os.path.dirname(os.path.abspath(__file__))
    path = [os.path.join(os.path.dirname(here), "regot-python_gb300"), here]
    r = subprocess.run([sys.executable, "-c", CODE % (path, solver)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    matrices = float(r.stdout.split("matrices")[1])
    # two, and the passes' partial sums (a few hundredths); three before
    assert 1.9 < matrices < 2.6
