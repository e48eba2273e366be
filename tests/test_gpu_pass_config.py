"""What regot_pass_config says is what runs: FP64 problems of up to 2^24 entries
have one configuration of their own, so nothing is tuned or forced there."""
import numpy as np
import pytest

from problems import erot_points

pytestmark = pytest.mark.gpu

regot = pytest.importorskip("regot")
from regot import _lib  # noqa: E402

ROW = 0  # REGOT_PASS_EROT_ROW
SMALL = 2  # the configuration of the small FP64 tiles


@pytest.fixture
def lib():
    lib = _lib.load()
    lib.regot_autotune_clear()
    yield lib
    lib.regot_force_pass_config(-1)
    lib.regot_autotune_clear()


def _config(lib, n, m, precision):
    return lib.regot_pass_config(_lib.context(0).handle, ROW, precision, n, m)


@pytest.mark.parametrize("forced", [-1, 0, 1])
def test_small_fp64_problems_have_their_own_configuration(lib, forced):
    lib.regot_force_pass_config(forced)
    run = max(forced, 0)
    for n, m in [(3, 2), (1000, 800), (4096, 4096), (2, 1 << 23)]:
        assert _config(lib, n, m, _lib.REGOT_PREC_FP64) == SMALL
        assert _config(lib, n, m, _lib.REGOT_PREC_MIXED) == run
    for n, m in [(4097, 4096), (8192, 8192)]:
        assert _config(lib, n, m, _lib.REGOT_PREC_FP64) == run


def test_autotune_records_what_it_can_choose(lib):
    ctx = _lib.context(0)
    ctx.check(lib.regot_autotune(ctx.handle, 300, 200, _lib.REGOT_PREC_FP64, 2))
    assert _lib.autotune_entries() == []
    ctx.check(lib.regot_autotune(ctx.handle, 300, 200, _lib.REGOT_PREC_MIXED, 2))
    rows = _lib.autotune_entries()
    assert rows and all(r[1] == "mixed" for r in rows)


def test_choices_of_smaller_classes_do_not_serve_large_fp64_problems(lib, tmp_path):
    # a table that holds configuration 1 for the FP64 classes below 24, whose
    # passes run in tiles of their own, and for class 26
    ctx = _lib.context(0)
    ctx.check(lib.regot_autotune(ctx.handle, 300, 200, _lib.REGOT_PREC_MIXED, 1))
    device = _lib.autotune_entries()[0][0]
    path = tmp_path / "table.tsv"
    lines = ["%s\tfp64\t%d\t%d\t1\t2.0\t1.0\n" % (device, op, c)
             for op in range(64) for c in (22, 23)]
    path.write_text("".join(lines))
    lib.regot_autotune_clear()
    lib.regot_autotune_load(str(path).encode())
    assert _config(lib, 4097, 4096, _lib.REGOT_PREC_FP64) == 0
    path.write_text("".join(line.replace("\t22\t1", "\t26\t1") for line in lines))
    lib.regot_autotune_clear()
    lib.regot_autotune_load(str(path).encode())
    assert _config(lib, 8192, 8192, _lib.REGOT_PREC_FP64) == 1
    assert _config(lib, 4097, 4096, _lib.REGOT_PREC_FP64) == 1  # within two classes


def test_forcing_changes_no_fp64_result(lib):
    M, a, b = erot_points(120, 90, seed=2, dtype=np.float64)
    P = regot.Problem(M, a, b, precision="fp64")
    gamma = np.full(209, 0.01)
    grads = []
    for cfg in (-1, 0, 1):
        lib.regot_force_pass_config(cfg)
        grads.append(P.erot_dual_obj_grad(0.1, gamma)[1])
    P.close()
    assert np.array_equal(grads[0], grads[1]) and np.array_equal(grads[0], grads[2])
