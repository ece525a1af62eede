"""Attention and its gradients at the edges of the tiles its batched products run on: one and several tiles
of queries, keys and head columns, ragged ones, widths that TMA cannot address, a tile for each SM and
many more, and gradients that share a launch or are wanted alone."""
import numpy as np
import pytest

import modelspec_b200 as M
from helpers import ProgramText, assert_kernel_close, run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wanted", ["QKV", "K", "V", "Q"])
@pytest.mark.parametrize("batch,q_len,k_len,heads,d", [(1, 1, 4, 1, 4), (3, 77, 77, 3, 33), (2, 64, 68, 2, 16), (40, 36, 200, 2, 24), (5, 300, 452, 2, 40),
                                                       (16, 128, 128, 2, 64), (32, 132, 136, 2, 8), (2, 512, 512, 2, 128), (1, 100, 257, 1, 64)])
def test_attention_at_tile_edges(device, batch, q_len, k_len, heads, d, wanted):
    r = np.random.default_rng(batch * q_len + k_len + d)
    values = lambda *shape: r.standard_normal(shape).astype(np.float32)
    h = heads * d
    p = ProgramText()
    q = p.input("q", "f32", [batch * q_len, h])
    k, v = (p.input(name, "f32", [batch * k_len, h]) for name in ("k", "v"))
    mask = p.input("mask", "f32", [batch, k_len])
    g = p.input("g", "f32", [batch * q_len, h])
    attr = "[heads = %d]" % heads
    outputs = [(p.op("Attention", [batch * q_len, h], [q, k, v, mask], attr=attr), batch * q_len * h)]
    for name in wanted:
        rows = batch * (q_len if name == "Q" else k_len)
        outputs.append((p.op("AttentionGrad" + name, [rows, h], [q, k, v, mask, g], attr=attr), rows * h))
    for value, _ in outputs:
        p.output(value)
    m = (np.arange(batch * k_len).reshape(batch, k_len) % 5 != 1).astype(np.float32)
    m[:, 0] = 1.0
    feed = {"q": values(batch * q_len, h), "k": values(batch * k_len, h), "v": values(batch * k_len, h), "mask": m,
            "g": values(batch * q_len, h)}
    res = run_both(device, p.text(), feed, outputs=outputs, flags=M.PLAN_NO_GRAPH)
    masked = np.repeat(m.reshape(-1) == 0.0, h)
    for (cpu, gpu), name in zip(res, "O" + wanted):
        assert_kernel_close(gpu, cpu, scale=np.abs(cpu).max(), what=name)
        if name in "KV":
            assert not gpu.reshape(-1)[masked].any() and not np.signbit(gpu.reshape(-1)[masked]).any(), "a masked key's row is +0"
