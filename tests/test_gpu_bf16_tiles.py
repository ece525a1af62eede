"""The bf16 product on tiles of one CTA and of pairs of CTAs (ragged edges, several bands of tiles, more
tiles than the device holds at a time) against float64 products of the same operands, and the products
of a mixed-precision step that share launches (projections as one launch, their input gradients summed
as one product, weight gradients as jobs, gelu and its gradient as the tile drains) against the f32
plan of the same run."""
import ctypes as C

import numpy as np
import pytest

import modelspec_b200 as M
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
