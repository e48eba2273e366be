"""Order of the block sums that the resident CG kernels exchange.

k_plan_cg (csrc/newton_plan.cuh) and k_schur_cg (csrc/schur_plan.cuh) pass sums
between blocks through numbered slots: ``publish(s, ...)`` writes this block's
part of slot s, ``total(s)`` reads every block's part. Blocks are ordered by the
barriers of all blocks alone, so a slot may be read only after a barrier that
follows its writing, and written again only after a barrier that follows its
last reading. The kernels are read as text: the calls before the loop, two turns
of it, and the calls behind it.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "regot-python_gb300", "csrc")
CALL = re.compile(r"(?<!auto )\b(publish|total)\((\d)|\b(bar\.wait)\(")


def _block(text, at):
    """End of the braced block that opens at or after `at`."""
    depth = 0
    for k in range(text.index("{", at), len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced braces")


def _calls(text):
    return [(k[1], int(k[2])) if k[1] else ("wait", -1) for k in CALL.finditer(text)]


def _violations(calls):
    phase, read, written, bad = 0, {}, {}, []
    for what, slot in calls:
        if what == "wait":
            phase += 1
        elif what == "publish":
            if read.get(slot, -1) >= phase:
                bad.append("slot %d is written in the phase that reads it" % slot)
            written[slot] = phase
        else:
            if written.get(slot, phase) >= phase:
                bad.append("slot %d is read in the phase that writes it" % slot)
            read[slot] = phase
    return bad


def test_the_rule_itself():
    good = [("publish", 1), ("wait", -1), ("total", 1), ("publish", 0), ("wait", -1), ("total", 0)]
    assert _violations(good) == []
    assert _violations([("publish", 0), ("wait", -1), ("total", 0), ("publish", 0)])
    assert _violations([("publish", 0), ("total", 0)])


@pytest.mark.parametrize("file,kernel", [("newton_plan.cuh", "k_plan_cg"),
                                         ("schur_plan.cuh", "k_schur_cg")])
def test_slots_are_rewritten_behind_a_barrier(file, kernel):
    with open(os.path.join(CSRC, file)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    start = text.index(" %s(" % kernel)
    body = text[start:_block(text, start)]
    loop = body.index("while (!s_stop)")
    end = _block(body, loop)
    pre, turn, post = _calls(body[:loop]), _calls(body[loop:end]), _calls(body[end:])
    # the lambdas' own definitions are not calls; the kernels make some of each
    assert {"publish", "total", "wait"} <= {c[0] for c in pre} and len(turn) >= 6
    for turns in (0, 1, 2, 3):
        assert _violations(pre + turns * turn + post) == []


@pytest.mark.parametrize("form", ["false", "true"])
def test_arriving_at_a_barrier_orders_the_block(form):
    """GridBarrier::arrive() (csrc/grid_sync.cuh) stands between a block's
    reading of its shared memory and its warps' next writing of it: in both
    forms all of the block's threads pass a barrier of the block before one of
    them goes on. The cluster's arrive instruction alone lets a warp go on
    while another still reads."""
    with open(os.path.join(CSRC, "grid_sync.cuh")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    start = text.index("struct GridBarrier<%s> {" % form)
    body = text[start:_block(text, start)]
    at = body.index("void arrive()")
    arrive = body[at:_block(body, at)]
    assert "__syncthreads();" in arrive
    assert arrive.index("__syncthreads();") < arrive.index("asm volatile")
