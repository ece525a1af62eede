"""What surrounds the launches of a step: inputs handed over through the staging slots (small ones
read from pinned memory by the step's first kernel, large ones copied ahead beside the step before),
losses published in their step's slot, values read back into memory that is not pinned, and the
update launch at the edges of its chunks."""
import numpy as np
import pytest

import adamw_reference as R
import modelspec_b200 as M
from helpers import ProgramText, assert_bits_equal
from test_adamw_written_order import run_gpu

pytestmark = pytest.mark.gpu


# One float, below and above the 64 KB that are read in place, ragged, and 2 MB.
@pytest.mark.parametrize("n", [1, 16384 - 64, 16384 + 1, 300001, 524288])
@pytest.mark.parametrize("flags", [M.PLAN_DEFAULT, M.PLAN_NO_GRAPH])
def test_every_step_runs_on_the_inputs_staged_for_it(device, n, flags):
    p = ProgramText()
    a = p.input("a", "f32", [n]); b = p.input("b", "f32", [n])
    p.output(p.op("Mse", [], [a, b]))
    plan = M.Plan(device, p.text(), flags=flags)
    try:
        plan.set_input("b", np.zeros(n, dtype=np.float32))
        want = []
        for k in range(20):
            if k % 5 != 4:  # every fifth step runs on what is staged already
                value = np.float32(1 + k % 7)
                plan.set_input("a", np.full(n, value, dtype=np.float32))
            plan.run()
            want.append(value * value)
            if k >= 3:
                assert plan.loss_of(k - 3) == want[k - 3], k
        plan.sync()
        assert [plan.loss_of(k) for k in range(12, 20)] == want[12:]
        assert all(0.0 < plan.step_ms(k) < 1000.0 for k in range(12, 20))
        total, steps = plan.elapsed_ms()
        assert steps == 20 and total > 0.0
    finally:
        plan.destroy()


# One float, below and above the 64 KB that are read in place (and the eight pinned slots one request), eight slots of
# 2 MB in all and one beyond, 8 MB; a plan of its own, and one that
# shares another's parameters and so reads in place whatever the size. Steps waited for one by one, then
# steps submitted behind one another, then waited for again, some on what is staged already.
@pytest.mark.parametrize("n", [1, 8192 - 64, 8192, 16384 + 1, 32768, 32768 + 64, 2100001])
@pytest.mark.parametrize("shared", [False, True])
def test_large_inputs_of_steps_waited_for_and_of_steps_behind_one_another(device, n, shared):
    p = ProgramText()
    a = p.input("a", "f32", [n]); b = p.input("b", "f32", [n])
    p.output(p.op("Mse", [], [a, b]))
    plans = [M.Plan(device, p.text())]
    if shared:
        plans.append(M.Plan(device, p.text(), shares=plans[0]))
    plan = plans[-1]
    r = np.random.default_rng(n)
    values = [r.standard_normal(n).astype(np.float32) for _ in range(6)]
    zeros = np.zeros(n, dtype=np.float32)
    mean_square = [float(np.mean(np.square(v, dtype=np.float64))) for v in values]
    try:
        plan.run()  # on nothing set: zeros
        want, k, last = [0.0], 1, 0.0
        assert plan.loss_of(0) == 0.0
        plan.set_input("b", zeros)
        for burst in (1, 1, 5, 1, 11, 2, 1):
            for _ in range(burst):
                if k % 4 != 3:
                    plan.set_input("a", values[k % 6])
                    last = mean_square[k % 6]
                plan.run()
                want.append(last)
                k += 1
            for j in range(max(k - burst, k - 8), k):
                assert abs(float(plan.loss_of(j)) - want[j]) <= 1e-6 * want[j], (j, burst)
    finally:
        for one in reversed(plans):
            one.destroy()


# Around the sizes where the copy into pageable memory starts to be staged, takes a second piece, a
# second thread, and ends inside a piece.
@pytest.mark.parametrize("n", [3, 65535, 65536, 262144 + 1, 3 * 262144, 4 * 262144 + 5, 20 * 262144 - 1])
def test_values_arrive_whole_in_pageable_memory(device, n):
    p = ProgramText()
    a = p.input("a", "f32", [n])
    out = p.op("Add", [n], [a, a])
    p.output(out)
    plan = M.Plan(device, p.text())
    try:
        for seed in range(2):
            x = np.random.default_rng(seed).standard_normal(n).astype(np.float32)
            plan.set_input("a", x)
            plan.run()
            assert_bits_equal(plan.value(out, n), x + x)
    finally:
        plan.destroy()


# Tensors shorter than a vector, around one 1,024-element chunk, and more elements than short
# chunks are used for.
@pytest.mark.parametrize("inputs,outputs", [(1, 1), (31, 33), (32, 32), (41, 25), (1111, 1101)])
def test_the_update_launch_at_the_edges_of_its_chunks(device, inputs, outputs):
    r = np.random.default_rng(inputs)
    rows = 4
    batches = [{"x": r.standard_normal(rows * inputs).astype(np.float32), "y": r.standard_normal(rows * outputs).astype(np.float32)}] * 4
    run_gpu(device, R.two_parameters(2, 4, rows, inputs, outputs), 4, batches=batches, check_steps=3)
