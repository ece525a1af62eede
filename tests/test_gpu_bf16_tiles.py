"""The bf16 product on tiles of one CTA and of pairs of CTAs (ragged edges, several bands of tiles, more
tiles than the device holds at a time) against float64 products of the same operands, and the products
of a mixed-precision step that share launches (projections as one launch, their input gradients summed
as one product, weight gradients as jobs, gelu and its gradient as the tile drains) against the f32
plan of the same run. gelu and its gradient are also held to float64, element by element."""
import ctypes as C

import numpy as np
import pytest

import modelspec_b200 as M
from helpers import ProgramText
from modelspec_b200 import models, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(8, 8, 8), (2200, 712, 200), (4096, 512, 128), (5000, 1032, 776), (12000, 2056, 320), (768, 3072, 4096), (712, 30528, 64)])
@pytest.mark.parametrize("form", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("half_out", [False, True])
def test_bf16_products_at_the_edges_of_their_tiles(device, m, n, k, form, half_out):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + 3 * n + 7 * k)
    a = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
    b = torch.randn((k, n), device="cuda", generator=gen).to(torch.bfloat16)
    a_t, b_t = form[0] == "t", form[1] == "t"
    d_a, d_b = (a.t() if a_t else a).contiguous(), (b.t() if b_t else b).contiguous()
    c = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16 if half_out else torch.float32)
    L = M.lib()
    need = L.msx_op_matmul_bf16_workspace(m, n, k)
    ws = torch.empty(max(need, 1), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    rc = L.msx_op_matmul_bf16(ptr(d_a), int(a_t), ptr(d_b), int(b_t), ptr(c), int(half_out), m, n, k, ptr(ws), need, ptr(status),
                              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == M.OK, L.msx_last_error(None)
    want, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    assert int(status.item()) == 0
    bound = 1e-5 + 1e-4 * size + (2.0 ** -8 * want.abs() if half_out else 0.0)
    assert bool(((c.double() - want).abs() <= bound).all())


# One k block a tile, so that a warp's rows below C (whose accumulator is zeros) come right behind the stores
# of the tile before: the zeros must not reach a slab that such a store still reads. Every run the same bits.
@pytest.mark.parametrize("m,n,k,form", [(2888, 34848, 32, "nn"), (656, 12064, 24, "nt"), (832, 30528, 64, "nt"), (5000, 12064, 32, "tn"), (72, 40064, 16, "nn")])
@pytest.mark.parametrize("half_out", [False, True])
def test_rows_below_the_result_leave_no_zeros_in_it(device, m, n, k, form, half_out):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + n)
    a = torch.randn((m, k), device="cuda", generator=gen).to(torch.bfloat16)
    b = torch.randn((k, n), device="cuda", generator=gen).to(torch.bfloat16)
    a_t, b_t = form[0] == "t", form[1] == "t"
    d_a, d_b = (a.t() if a_t else a).contiguous(), (b.t() if b_t else b).contiguous()
    want, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    bound = 1e-5 + 1e-4 * size + (2.0 ** -8 * want.abs() if half_out else 0.0)
    L = M.lib()
    need = L.msx_op_matmul_bf16_workspace(m, n, k)
    ws = torch.empty(max(need, 1), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    for _ in range(12):
        c = torch.full((m, n), float("nan"), device="cuda", dtype=torch.bfloat16 if half_out else torch.float32)
        torch.cuda.synchronize()
        rc = L.msx_op_matmul_bf16(ptr(d_a), int(a_t), ptr(d_b), int(b_t), ptr(c), int(half_out), m, n, k, ptr(ws), need, ptr(status),
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == M.OK, L.msx_last_error(None)
        assert bool(((c.double() - want).abs() <= bound).all())
    assert int(status.item()) == 0


@pytest.mark.parametrize("shape", [dict(batch=3, seq=24, hidden=48, heads=2, ffn=72), dict(batch=11, seq=200, hidden=200, heads=5, ffn=712),
                                   dict(batch=40, seq=128, hidden=512, heads=8, ffn=2048)])
def test_products_that_share_launches_against_the_f32_plan(device, shape):
    vocab, steps = 1000, 3
    source = models.bert(layers=2, vocab=vocab, lr=1e-3, warmup_steps=1, steps=steps, dropout=0.1, **shape)
    masked = models.default_masked_rows(shape["batch"] * shape["seq"])
    runs = [M.Training(device, source, masked, flags) for flags in (M.PLAN_DEFAULT, M.PLAN_BF16)]
    try:
        for k in range(steps):
            losses = []
            for run in runs:
                for name, value in synthetic.mlm_batch(k, vocab=vocab, seq=shape["seq"], batch=shape["batch"]).items():
                    run.set_input(name, value)
                run.step(k, steps + 1)
                losses.append(float(run.loss()))
            assert abs(losses[0] - losses[1]) <= 2e-2 * abs(losses[0]), losses
        for i, (path, _) in enumerate(runs[0].step_plan.params()):
            if path.endswith("_bk"):
                continue  # its exact gradient is 0
            want, got = (run.step_plan.moment_download(i, "m") for run in runs)
            assert np.linalg.norm(got - want) <= 6e-2 * np.linalg.norm(want) + 1e-12, path
    finally:
        for run in runs:
            run.destroy()


# One CTA and pairs, ragged rows and columns, several bands of tiles, more tiles than the device holds. The three
# values are read through products with the identity, which are exact; the product in front of gelu_grad is not
# stored, so its rounding to bf16 is in the bound: 2^-8 of the value for a rounding that fell the other way, and the
# kernel tolerance of the f32 sum.
@pytest.mark.parametrize("m,n,k", [(100, 72, 40), (200, 200, 48), (2200, 712, 200), (5000, 1032, 136), (4096, 3072, 768)])
def test_every_element_of_gelu_and_its_gradient_as_a_tile_drains(device, m, n, k):
    import torch
    p = ProgramText()
    k2 = k + 8  # a shape of its own: products of one shape would share a launch without an epilogue
    sizes = {"t1": (m, k), "t2": (m, k2), "w1": (k, n), "w2": (k2, n), "eye": (n, n)}
    at = {name: p.param(name, list(shape)) for name, shape in sizes.items()}
    bias = p.param("bias", [n])
    ids = p.input("ids", "i32", [m])
    x, x2 = p.op("Embedding", [m, k], [at["t1"], ids]), p.op("Embedding", [m, k2], [at["t2"], ids])
    z = p.op("AddRows", [m, n], [p.op("MatMul", [m, n], [x, at["w1"]]), bias])
    y = p.op("Gelu", [m, n], [z])
    d = p.op("GeluGrad", [m, n], [z, p.op("MatMul", [m, n], [x2, at["w2"]])])
    outputs = [p.op("MatMul", [m, n], [value, at["eye"]]) for value in (z, y, d)]
    for value in outputs:
        p.output(value)
    plan = M.Plan(device, p.text(), flags=M.PLAN_BF16)
    try:
        kernels = [plan_kernel for plan_kernel, _, _, _ in plan.profile_step()]
        assert "matmul" in kernels and not any("gelu" in name for name in kernels), kernels
        gen = torch.Generator(device="cuda").manual_seed(m + n + k)
        half = {name: (torch.randn(shape, device="cuda", generator=gen) * (2.0 if name == "t1" else 1.0) * shape[0] ** (-0.5 if name[0] == "w" else 0.0)).to(torch.bfloat16)
                for name, shape in sizes.items() if name != "eye"}
        half["eye"] = torch.eye(n, device="cuda").to(torch.bfloat16)
        b = torch.randn(n, device="cuda", generator=gen)
        for i, (path, _) in enumerate(plan.params()):
            plan.param_upload(i, (b if path == "bias" else half[path].float()).cpu().numpy())
        plan.set_input("ids", np.arange(m, dtype=np.int32))
        plan.run()
        got_z, got_y, got_d = (torch.from_numpy(plan.value(value, m * n)).cuda().double().reshape(m, n) for value in outputs)
        f = {name: value.double() for name, value in half.items()}
        want_z, size = f["t1"] @ f["w1"] + b.double(), f["t1"].abs() @ f["w1"].abs() + b.double().abs()
        assert bool(((got_z - want_z).abs() <= 2.0 ** -8 * want_z.abs() + 1e-5 + 1e-4 * size).all())
        # Of the stored argument.
        u = 0.7978845608028654 * (got_z + 0.044715 * got_z ** 3)
        s = torch.sigmoid(2.0 * u)
        slope = s + got_z * s * (1.0 - s) * 2.0 * 0.7978845608028654 * (1.0 + 3.0 * 0.044715 * got_z ** 2)
        want_y = got_z * s
        assert bool(((got_y - want_y).abs() <= 2.0 ** -8 * want_y.abs() + 1e-6).all())
        g, size = f["t2"] @ f["w2"], f["t2"].abs() @ f["w2"].abs()
        bound = slope.abs() * (2.0 ** -8 * g.abs() + 1e-5 + 1e-4 * size) + 2.0 ** -8 * (slope * g).abs() + 1e-6 * (1.0 + g.abs())
        assert bool(((got_d - slope * g).abs() <= bound).all())
    finally:
        plan.destroy()
