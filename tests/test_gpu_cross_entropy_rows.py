"""The cross-entropy with its gradient on logits as a plan stores them (rows padded to 16 bytes), in
both storage types, at the edges of each kernel's range: a warp a row up to 1,024 logits, then 128 to
1,024 threads a row, the row's last piece partly or wholly inside it."""
import numpy as np
import pytest

import modelspec_b200 as M
from helpers import ProgramText

pytestmark = pytest.mark.gpu

EDGES = [1, 3, 10, 128, 129, 1009, 1024, 1025, 4096, 4099, 8192, 8201, 16384, 16391, 30522, 32768, 32777, 50001]


@pytest.mark.parametrize("flags", [M.PLAN_DEFAULT, M.PLAN_BF16], ids=["f32", "bf16"])
@pytest.mark.parametrize("v", EDGES)
@pytest.mark.parametrize("rows", [8, 136])
def test_padded_rows_against_float64(device, rows, v, flags):
    if rows > 8 and v > 5000 and v % 2 == 0:
        pytest.skip("the long rows' edges are covered with few rows")
    half = flags == M.PLAN_BF16
    if half and v < 8:
        pytest.skip("a mixed-precision plan stores no rows of fewer than 8 elements")
    r = np.random.default_rng(rows * 100003 + v)
    p = ProgramText()
    ids = p.input("ids", "i32", [rows]); labels = p.input("labels", "i32", [rows]); w = p.input("w", "f32", [rows])
    unit = p.param("unit", [rows, rows]); table = p.param("table", [v, rows])
    one = p.node("Tensor<f32, []>", "Scalar 1.0")
    a = p.op("Embedding", [rows, rows], [unit, ids])
    logits = p.op("MatMul", [rows, v], [a, p.op("Transpose", [rows, v], [table])])
    loss = p.op("CrossEntropy", [], [logits, labels, w]); d = p.op("CrossEntropyGrad", [rows, v], [logits, labels, w, one])
    at = p.op("Transpose", [rows, rows], [a]); back = p.op("MatMul", [rows, v], [at, d])
    p.output(loss); p.output(back)
    # The identity around the cross-entropy: the logits are the table, what comes back is the gradient.
    x = (r.standard_normal((rows, v)) * 4).astype(np.float32)
    x = (x.view(np.uint32) & np.uint32(0xffff0000)).view(np.float32)  # values that bf16 holds
    x[0, :] = 0.0
    wv = (r.random(rows) < 0.6).astype(np.float32)
    wv[0], wv[-1] = 1.0, 0.5
    yv = r.integers(0, v, size=rows).astype(np.int32)
    yv[0], yv[-1] = v - 1, 0
    plan = M.Plan(device, p.text(), flags=flags | M.PLAN_NO_GRAPH | M.PLAN_GUARD)
    try:
        plan.set_input("ids", np.arange(rows, dtype=np.int32)); plan.set_input("labels", yv); plan.set_input("w", wv)
        plan.param_upload(0, np.eye(rows, dtype=np.float32)); plan.param_upload(1, np.ascontiguousarray(x.T))
        for _ in range(2):  # the second run finds the arrival counter as the first left it
            plan.run(); plan.sync(); plan.check_guards()
            got_loss, got = float(plan.value(loss, 1)[0]), plan.value(back, rows * v).reshape(rows, v).astype(np.float64)
    finally:
        plan.destroy()
    x64 = x.astype(np.float64)
    top = x64.max(axis=1, keepdims=True)
    e = np.exp(x64 - top)
    prob = e / e.sum(axis=1, keepdims=True)
    target = np.zeros_like(prob); target[np.arange(rows), yv] = 1.0
    scale = (wv.astype(np.float64) / wv.sum())[:, None]
    want = scale * (prob - target)
    nll = np.log(e.sum(axis=1)) + top[:, 0] - x64[np.arange(rows), yv]
    # Each probability to a few units of its f32 arithmetic on arguments of up to 40 (the hardware's exponential: 2^-21
    # relative, its argument rounded to 40 * 2^-24), the stored gradient and its product to bf16's half unit.
    bound = scale * (1e-5 * prob + 2.0 ** -21) + (2.0 ** -8 if half else 1e-6) * np.abs(want)
    off = np.abs(got - want)
    assert (off <= bound).all(), "%d of %d outside; worst %g of its bound" % ((off > bound).sum(), off.size, (off / np.maximum(bound, 1e-300)).max())
    assert not got[wv == 0.0].any()
    assert abs(got_loss - (wv * nll).sum() / wv.sum()) <= 1e-5 * max(1.0, abs(nll).max())
