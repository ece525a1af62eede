"""relu, gelu and their gradients inside the f32 product whose result they take (the FMA tiles, with and without a cluster, and
the 64-row tiles 32, 64 and 128 wide, with rows on and off 16 bytes): the bits of the launches of their own, which a program gets
whose product is an output."""
import numpy as np
import pytest

import modelspec_b200 as M
from helpers import ProgramText, assert_bits_equal

pytestmark = pytest.mark.gpu


def program(m, n, k, act, bias, apart):
    p = ProgramText()
    x = p.input("x", "f32", [m, k]); g = p.input("g", "f32", [m, k + 4]); w = p.param("w", [k, n]); v = p.param("v", [k + 4, n]); b = p.param("b", [n])
    before = p.op("MatMul", [m, n], [x, w])
    before = p.op("AddRows", [m, n], [before, b]) if bias else before
    after = p.op(act, [m, n], [before])
    adjoint = p.op("MatMul", [m, n], [g, v])
    back = p.op(act + "Grad", [m, n], [before, adjoint])
    ends = [p.op("Add", [m, n], [after, after]), p.op("Add", [m, n], [back, back])]
    for value in ends + ([before, adjoint] if apart else []):
        p.output(value)
    return p.text(), ends


@pytest.mark.parametrize("act", ["Relu", "Gelu"])
@pytest.mark.parametrize("m,n,k,bias", [(1, 1, 1, True), (33, 31, 17, False), (64, 128, 784, True), (5, 7, 300, True), (385, 250, 99, True), (700, 250, 99, False),
                                        (1500, 130, 250, True), (64, 66, 2000, True), (900, 33, 130, False), (1500, 128, 249, True), (1500, 512, 249, False),
                                        (1500, 2048, 249, True)])
def test_an_activation_inside_a_product_has_the_bits_of_its_own_launch(device, m, n, k, bias, act):
    r = np.random.default_rng(m * 1000 + n)
    x, g = (r.standard_normal((m, depth)).astype(np.float32) for depth in (k, k + 4))  # (of one shape they would share a launch)
    w, v = (r.standard_normal((depth, n)).astype(np.float32) / np.float32(np.sqrt(k)) for depth in (k, k + 4))
    b = r.standard_normal(n).astype(np.float32)
    results, launches = [], []
    for apart in (False, True):
        text, ends = program(m, n, k, act, bias, apart)
        listed = [line.split(": ")[1].split()[0] for line in M.schedule_describe(text).splitlines() if ": " in line]
        launches.append((listed.count("matmul"), sum(kernel.startswith((act.lower(), "unary")) for kernel in listed)))
        plan = M.Plan(device, text, flags=M.PLAN_NO_GRAPH | M.PLAN_GUARD)
        try:
            plan.set_input("x", x); plan.set_input("g", g)
            for at, value in enumerate((w, v, b)[: 3 if bias else 2]):
                plan.param_upload(at, value)
            plan.run(); plan.sync(); plan.check_guards()
            results.append([plan.value(e, m * n) for e in ends])
        finally:
            plan.destroy()
    assert launches == [(2, 0), (2, 2)], "the activation and its gradient: inside the products, and apart"
    for name, inside, own in zip((act, act + "Grad"), *results):
        assert_bits_equal(inside, own, name)
    z = x.astype(np.float64) @ w.astype(np.float64) + (b if bias else 0.0)
    want = np.maximum(z, 0.0) if act == "Relu" else z / (1 + np.exp(-2 * np.sqrt(2 / np.pi) * (z + 0.044715 * z ** 3)))
    assert np.abs(results[0][0].reshape(m, n) / 2 - want).max() <= 1e-4 * max(1.0, np.abs(want).max())
