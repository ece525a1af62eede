"""The f32 product at the edges of its kernels: the FMA tiles (one CTA a tile, and clusters that share a
tile's k), the TMA-fed tiles of one CTA and of pairs of CTAs, sums that leave tensor memory several
times, results TMA cannot store, more tiles than the device holds. Against float64 products of the
same operands: |g - c| <= 6e-6 sum |a||b| up to k = 1,024 and 2e-5 beyond, which the sums of a
truncating accumulator left to run would exceed (6e-5 at k = 3,076)."""
import ctypes as C

import pytest

import modelspec_b200 as M

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (33, 17, 31), (64, 10, 128), (64, 128, 784), (100, 37, 1500), (385, 99, 250), (700, 60, 2048),  # FMA, clusters
          (2048, 96, 160), (4096, 128, 512), (3000, 200, 100), (4096, 512, 128), (2100, 516, 772),                   # one CTA
          (16384, 768, 800), (5000, 1028, 3076), (300, 30522, 1600), (1300, 4001, 100),                              # pairs, segments, odd rows
          (92, 17609, 2207), (1567, 1162, 4455), (25, 32, 2217), (1261, 27, 899)]                                   # 64-row tiles of each width, split and not


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("form", ["nn", "nt", "tn", "tt"])
def test_f32_products_at_the_edges_of_their_kernels(device, m, n, k, form):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + 3 * n + 7 * k)
    # Mostly one sign: a bias of the sums shows.
    a = torch.randn((m, k), device="cuda", generator=gen) + 0.5
    b = torch.randn((k, n), device="cuda", generator=gen) + 0.5
    a_t, b_t = form[0] == "t", form[1] == "t"
    d_a, d_b = (a.t() if a_t else a).contiguous(), (b.t() if b_t else b).contiguous()
    c = torch.full((m, n), float("nan"), device="cuda")
    L = M.lib()
    need = L.msx_op_matmul_workspace(m, n, k)
    ws = torch.empty(max(need, 1), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    rc = L.msx_op_matmul(ptr(d_a), int(a_t), ptr(d_b), int(b_t), ptr(c), m, n, k, ptr(ws), need, ptr(status),
                         C.c_void_p(torch.cuda.current_stream().cuda_stream), 0)
    assert rc == M.OK, L.msx_last_error(None)
    want = a.double() @ b.double()
    size = a.double().abs() @ b.double().abs()
    off = c.double() - want
    assert int(status.item()) == 0
    worst = float((off.abs() / size).max())
    assert worst <= (6e-6 if k <= 1024 else 2e-5), worst


# Weight gradients as deep as a batch has rows: on pairs of CTAs (unsplit and split) and on tiles of one
# CTA. What truncates is a segment of 96 k slices in tensor memory, three MMAs a slice, each at most
# 2^-23 of a sum that grows to the segment's: 96 * 3 * 2^-23 / 2 = 1.7e-5 of sum |a||b| if every MMA lost
# a whole unit in the last place, half of it on average (a sum of 256 k blocks was 2.8e-5 low). The last two have rows TMA cannot address: a
# sum of 85 k blocks on the 64-row tiles was 9.0e-6 low.
@pytest.mark.parametrize("m,n,k", [(768, 3072, 16384), (3072, 768, 16384), (768, 768, 16384), (396, 1024, 60000), (96, 64, 20000), (4096, 260, 9001),
                                   (429, 1281, 16384), (771, 771, 32001), (1567, 1162, 4455), (33, 29, 200001)])
def test_deep_weight_gradients_do_not_come_out_low(device, m, n, k):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(m + 3 * n + 7 * k)
    a = torch.randn((k, m), device="cuda", generator=gen) + 0.5
    b = torch.randn((k, n), device="cuda", generator=gen) + 0.5
    c = torch.full((m, n), float("nan"), device="cuda")
    L = M.lib()
    need = L.msx_op_matmul_workspace(m, n, k)
    ws = torch.empty(max(need, 1), device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())
    torch.cuda.synchronize()
    rc = L.msx_op_matmul(ptr(a), 1, ptr(b), 0, ptr(c), m, n, k, ptr(ws), need, ptr(status), C.c_void_p(torch.cuda.current_stream().cuda_stream), 0)
    assert rc == M.OK, L.msx_last_error(None)
    size = a.double().abs().t() @ b.double().abs()
    off = (c.double() - a.double().t() @ b.double()).abs()
    assert int(status.item()) == 0
    worst = float((off / size).max())
    assert worst <= 8.6e-6, worst
