"""Column sums that a step leaves for its finalize launch: widths around the 128 columns from which a lane reads four
of them (127 and 130 stay one by one), row counts around a chunk's 128, several matrices of both kinds in one launch,
and one large enough for a launch of its own. Against float64: a sum of n terms in any order is within n * 2^-24 of
its magnitudes' sum, and a bf16 plan rounds each term by 2^-8 of it at most before that."""
import numpy as np
import pytest

import modelspec_b200 as M
from helpers import ProgramText

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("rows,widths", [(1, [128]), (127, [32, 128, 136]), (129, [256, 24, 640]), (300, [127, 130, 132, 1032]), (6600, [640])])
def test_column_sums_left_for_the_finalize_launch(device, rows, widths, half):
    if half:
        widths = [w + -w % 8 for w in widths]
    r = np.random.default_rng(rows + len(widths))
    p = ProgramText()
    ids = p.input("ids", "i32", [rows])
    # Rows of a table: a bf16 plan stores what an op computes as bf16, an input not.
    terms = [p.op("Embedding", [rows, w], [p.param("t%d" % k, [rows, w]), ids]) for k, w in enumerate(widths)]
    sums = [p.op("SumRows", [w], [t]) for t, w in zip(terms, widths)]
    for s in sums:
        p.output(s)
    flags = M.PLAN_BF16 if half else M.PLAN_DEFAULT
    plan = M.Plan(device, p.text(), flags=flags)
    feed = [np.abs(r.standard_normal((rows, w))).astype(np.float32) for w in widths]
    for k, g in enumerate(feed):
        plan.param_upload(k, g)
    plan.set_input("ids", r.permutation(rows).astype(np.int32))
    kernels = [line.split()[1] for line in M.schedule_describe(p.text(), flags).strip().splitlines()[:-1]]
    assert kernels[len(widths):] == ["sum_rows" if rows == 6600 else "sum_rows_batched", "finalize_sums"], kernels
    plan.run()
    plan.sync()
    for s, g, w in zip(sums, feed, widths):
        exact = g.astype(np.float64).sum(0)
        bound = exact * (rows * 2.0**-24 + (2.0**-8 if half else 0.0))
        assert (np.abs(plan.value(s, w) - exact) <= bound).all()
    plan.destroy()
