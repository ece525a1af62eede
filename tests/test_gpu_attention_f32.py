"""f32 attention with the scores on the chip, forward and gradients, element by element against float64 at the edges
of its tiles: one query or key, 128 and one more of both, key tiles of 64 and 128 that end inside, heads that no 16-byte
access fits, tiles whose keys are all masked."""
import ctypes as C

import numpy as np
import pytest

import modelspec_b200 as M
from helpers import ProgramText

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1, 1), (2, 77, 77, 3, 33), (2, 128, 128, 2, 64), (1, 129, 130, 2, 40), (2, 16, 512, 1, 8), (1, 200, 65, 2, 64), (3, 64, 64, 2, 32),
          (1, 300, 257, 1, 20), (1, 130, 512, 2, 61), (2, 33, 16, 5, 16), (1, 5, 385, 1, 64), (1, 256, 17, 1, 31)]


def program(batch, q_len, k_len, heads, d, wanted):
    h = heads * d
    p = ProgramText()
    q = p.input("q", "f32", [batch * q_len, h]); k = p.input("k", "f32", [batch * k_len, h])
    v = p.input("v", "f32", [batch * k_len, h]); mask = p.input("mask", "f32", [batch, k_len])
    g = p.input("g", "f32", [batch * q_len, h])
    attr = "[heads = %d]" % heads
    values = {"O": (p.op("Attention", [batch * q_len, h], [q, k, v, mask], attr=attr), q_len)}
    for name in wanted:
        rows = q_len if name == "Q" else k_len
        values[name] = (p.op("AttentionGrad" + name, [batch * rows, h], [q, k, v, mask, g], attr=attr), rows)
    for value, _ in values.values():
        p.output(value)
    return p.text(), values


def float64(feed, batch, q_len, k_len, heads, d):
    """The op and its gradients, and for each what the arithmetic of 11 + 11 bit operands and f32 sums can be off by."""
    eps = 2.0 ** -20
    split = lambda x, rows: x.astype(np.float64).reshape(batch, rows, heads, d).transpose(0, 2, 1, 3)
    q, k, v, g = split(feed["q"], q_len), split(feed["k"], k_len), split(feed["v"], k_len), split(feed["g"], q_len)
    kT, vT = k.transpose(0, 1, 3, 2), v.transpose(0, 1, 3, 2)
    scale = 1.0 / np.sqrt(d)
    s = q @ kT * scale
    off_p = eps * (4 + (np.abs(q) @ np.abs(kT) * scale).max(axis=-1, keepdims=True))  # of itself
    s = np.where(feed["mask"][:, None, None, :] != 0, s, -np.inf)
    p = np.exp(s - s.max(axis=-1, keepdims=True))
    p /= p.sum(axis=-1, keepdims=True)
    out = p @ v
    off_out = (2 * off_p + eps) * (p @ np.abs(v))
    dP = g @ vT
    dot = (out * g).sum(axis=-1, keepdims=True)
    dS = p * (dP - dot) * scale
    off_dP = eps * (np.abs(g) @ np.abs(vT)) + (off_out * np.abs(g)).sum(axis=-1, keepdims=True) + eps * (np.abs(out * g)).sum(axis=-1, keepdims=True)
    off_dS = scale * p * (off_dP + 2 * off_p * (np.abs(dP) + np.abs(dot)))
    T = lambda x: x.transpose(0, 1, 3, 2)
    join = lambda x: x.transpose(0, 2, 1, 3).reshape(-1)
    want = {"O": out, "Q": dS @ k, "K": T(dS) @ q, "V": T(p) @ g}
    off = {"O": off_out, "Q": off_dS @ np.abs(k) + eps * (np.abs(dS) @ np.abs(k)), "K": T(off_dS) @ np.abs(q) + eps * (T(np.abs(dS)) @ np.abs(q)),
           "V": T(2 * off_p * p) @ np.abs(g) + eps * (T(p) @ np.abs(g))}
    return {n: (join(want[n]), join(off[n])) for n in want}


def feed_of(batch, q_len, k_len, heads, d):
    r = np.random.default_rng(q_len * 1000 + k_len + d)
    draw = lambda rows: r.standard_normal((batch * rows, heads * d)).astype(np.float32)
    feed = {"q": 2 * draw(q_len), "k": draw(k_len), "v": draw(k_len), "g": draw(q_len)}
    mask = (r.random((batch, k_len)) < 0.8).astype(np.float32)
    mask[0, : k_len - 1] = 0.0  # every tile but the last has no key of this sequence
    mask[:, k_len - 1] = 1.0
    feed["mask"] = mask
    return feed


def check(got, feed, shape):
    want = float64(feed, *shape)
    for name in got:
        value, off = want[name]
        bad = ~(np.abs(got[name] - value) <= off + 1e-30)
        assert not bad.any(), "%s: %d of %d outside; worst %g of its bound" % (
            name, bad.sum(), bad.size, (np.abs(got[name] - value) / np.maximum(off, 1e-300)).max())
    masked = np.repeat(feed["mask"].reshape(-1) == 0.0, shape[3] * shape[4])
    for name in set("KV") & set(got):
        assert not got[name][masked].any() and not np.signbit(got[name][masked]).any()


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("wanted", ["QKV", "V", "QK"])
@pytest.mark.parametrize("batch,q_len,k_len,heads,d", SHAPES)
def test_every_element_of_the_kernels_against_float64(device, batch, q_len, k_len, heads, d, wanted, shift):
    """`shift`: every operand a float behind a 16-byte boundary."""
    if (wanted != "QKV" or shift) and (q_len, d) not in [(77, 33), (129, 40), (128, 64)]:
        pytest.skip("some of the gradients, and unaligned operands: three shapes")
    import torch
    shape = (batch, q_len, k_len, heads, d)
    feed = feed_of(*shape)
    kept = []

    def buffer(count, value=None):
        t = torch.full((count + 8,), float("nan"), dtype=torch.float32, device="cuda")
        if value is not None:
            t[shift : shift + count] = torch.from_numpy(value.reshape(-1)).cuda()
        kept.append(t)
        return t[shift : shift + count]

    ptr = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None
    operand = {n: buffer(v.size, v) for n, v in feed.items()}
    rows = {"O": q_len, "Q": q_len, "K": k_len, "V": k_len}
    out = {n: buffer(batch * rows[n] * heads * d) for n in "O" + wanted}
    p = buffer(batch * heads * q_len * k_len) if k_len <= 128 else None
    stats, status = torch.zeros(2 * batch * heads * q_len, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    rc = M.lib().msx_op_attention_f32(ptr(operand["q"]), ptr(operand["k"]), ptr(operand["v"]), ptr(operand["mask"]), ptr(operand["g"]), ptr(out["O"]),
                                      ptr(out.get("Q")), ptr(out.get("K")), ptr(out.get("V")), ptr(stats), ptr(p), *shape, ptr(status), None)
    assert rc == M.OK, M.lib().msx_last_error(None).decode()
    torch.cuda.synchronize()
    assert int(status.item()) == 0, "a bounded wait inside a kernel ran out"
    check({n: t.cpu().numpy().astype(np.float64) for n, t in out.items()}, feed, shape)
    for t in kept:  # nothing outside of an operand was written
        assert torch.isnan(t[:shift]).all() and torch.isnan(t[-(8 - shift):]).all()
    # The statistics are pairs: refused where no pair can be stored.
    assert M.lib().msx_op_attention_f32(ptr(operand["q"]), ptr(operand["k"]), ptr(operand["v"]), ptr(operand["mask"]), ptr(operand["g"]), ptr(out["O"]),
                                        ptr(out.get("Q")), ptr(out.get("K")), ptr(out.get("V")), C.c_void_p(stats.data_ptr() + 4), ptr(p), *shape,
                                        ptr(status), None) == M.BAD_ARGUMENT
    if p is not None:
        sums = p.cpu().numpy().astype(np.float64).reshape(-1, k_len).sum(axis=1)
        assert np.abs(sums - 1.0).max() <= 1e-5


# The halves of an operand stay finite up to the largest float: rounding to the nearest would take what lies within 2^-11 of it to
# infinity, and its remainder with it.
@pytest.mark.parametrize("batch,q_len,k_len,heads,d", [(1, 33, 16, 2, 16), (1, 130, 300, 1, 64)])
def test_values_next_to_the_largest_float(device, batch, q_len, k_len, heads, d):
    import torch
    shape = (batch, q_len, k_len, heads, d)
    feed = feed_of(*shape)
    feed["mask"][:] = 0.0
    feed["mask"][:, 3] = 1.0  # one key: its probability is 1, and O the row of V itself
    # A result is off by up to 2^-20 of itself (float64 above): as far below the largest float as that, it is finite.
    largest = np.float32(3.4028235e38)
    feed["v"][:] = np.where(np.random.default_rng(0).random(feed["v"].shape) < 0.5, -largest * np.float32(1 - 2.0 ** -13), largest * np.float32(1 - 2.0 ** -19))
    operand = {n: torch.from_numpy(x.reshape(-1)).cuda() for n, x in feed.items()}
    out, status = torch.zeros(batch * q_len * heads * d, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    rc = M.lib().msx_op_attention_f32(ptr(operand["q"]), ptr(operand["k"]), ptr(operand["v"]), ptr(operand["mask"]), None, ptr(out), None, None, None, None,
                                      None, *shape, ptr(status), None)
    assert rc == M.OK and int(status.item()) == 0
    want = np.repeat(feed["v"].reshape(batch, 1, k_len, heads * d)[:, :, 3], q_len, axis=1).reshape(-1)
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    assert np.abs(got.astype(np.float64) / want - 1.0).max() <= 2.0 ** -20


# One way each: both kernels, the forward with its probabilities left for the gradients' products (rows on and off 16 bytes),
# neither. Which way a plan takes shows in what its gradients read (the statistics and O, or probabilities), and in the bits of O.
@pytest.mark.parametrize("batch,q_len,k_len,heads,d,way", [(32, 128, 128, 2, 64, "both"), (5, 77, 77, 3, 33, "both"), (32, 100, 100, 8, 32, "forward"),
                                                          (60, 96, 99, 6, 7, "forward"), (2, 160, 256, 3, 16, "products")])
def test_a_plan_takes_each_way(device, batch, q_len, k_len, heads, d, way):
    import torch
    shape = (batch, q_len, k_len, heads, d)
    feed = feed_of(*shape)
    text, values = program(*shape, "QKV")
    backward = next(line for line in M.schedule_describe(text).splitlines() if " attention_backward " in line)
    assert (" %%%d " % values["O"][0] in backward.split("writes")[0]) == (way == "both"), backward
    plan = M.Plan(device, text, flags=M.PLAN_NO_GRAPH | M.PLAN_GUARD)
    try:
        for name, value in feed.items():
            plan.set_input(name, value)
        plan.run(); plan.sync(); plan.check_guards()
        got = {name: plan.value(at, batch * rows * heads * d) for name, (at, rows) in values.items()}
        check(got, feed, shape)
    finally:
        plan.destroy()
    operand = {n: torch.from_numpy(x.reshape(-1)).cuda() for n, x in feed.items()}
    out, status = torch.zeros(batch * q_len * heads * d, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    rc = M.lib().msx_op_attention_f32(ptr(operand["q"]), ptr(operand["k"]), ptr(operand["v"]), ptr(operand["mask"]), None, ptr(out), None, None, None, None,
                                      None, *shape, ptr(status), None)
    assert rc == M.OK and int(status.item()) == 0
    assert (out.cpu().numpy().tobytes() == np.ascontiguousarray(got["O"]).tobytes()) == (way != "products")
