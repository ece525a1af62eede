"""Inputs that the host loop writes straight into the slot their step reads: a run that sets only what changed is, bit
for bit, the run that sets everything; what reads the batch beside the step sees it as it was last set."""
import numpy as np
import pytest

import modelspec_b200 as M
from helpers import assert_bits_equal
from modelspec_b200 import models

pytestmark = pytest.mark.gpu

STEPS = 21  # more than twice the slots


# Below and above the 64 KB of inputs that a step reads in place.
@pytest.mark.parametrize("batch,inputs", [(8, 20), (64, 300)])
def test_a_run_that_sets_only_what_changed(device, batch, inputs):
    source = models.mlp_classifier(batch=batch, inputs=inputs, hidden=16, classes=5, steps=STEPS)
    r = np.random.default_rng(batch)
    x = [r.random((batch, inputs), dtype=np.float32) for _ in range(STEPS)]
    y = [r.integers(0, 5, batch, dtype=np.int32) for _ in range(STEPS)]
    ones = np.ones(batch, dtype=np.float32)
    whole, sparse = M.Training(device, source), M.Training(device, source)
    try:
        now = {}
        losses = []
        for k in range(STEPS):
            new = {"x": x[k]} if k in (0, 1, 2, 13) else {}
            if k in (0, 2, 3, 4, 5):
                new["labels"] = y[k]
            if k == 0:
                new["weights"] = ones
            now.update(new)
            for run, values in ((whole, now), (sparse, new)):
                for name, value in values.items():
                    run.set_input(name, value)
                run.step(k, STEPS)
            losses.append((whole.loss_of(k), sparse.loss_of(k)))
            if k in (3, 12):
                # In the middle of a batch's setting, and by every other reader of it.
                for run in (whole, sparse):
                    run.set_input("labels", y[7])
                    assert_bits_equal(run.get_input("x", batch * inputs), now["x"].reshape(-1))
                    assert (run.get_input("labels", batch, np.int32) == y[7]).all()
                a, b = whole.infer(), sparse.infer()
                assert_bits_equal(a[0], b[0]); assert a[1] == b[1] == whole.final_loss() == sparse.final_loss()
                for run in (whole, sparse):
                    run.set_input("labels", now["labels"])
        for a, b in losses:
            assert a == b
        for i in range(4):
            assert_bits_equal(sparse.step_plan.param_download(i), whole.step_plan.param_download(i))
    finally:
        whole.destroy(); sparse.destroy()


def test_a_bad_batch_is_refused_by_its_step_and_the_run_goes_on(device):
    source = models.mlp_classifier(batch=8, inputs=12, hidden=16, classes=5, steps=8)
    r = np.random.default_rng(1)
    x, y = r.random((8, 12), dtype=np.float32), r.integers(0, 5, 8, dtype=np.int32)
    good, bad = M.Training(device, source), M.Training(device, source)
    try:
        for k in range(4):
            for run in (good, bad):
                run.set_input("x", x + k); run.set_input("labels", y); run.set_input("weights", np.ones(8, dtype=np.float32))
            if k >= 2:
                bad.set_input("labels", y + 5)  # accepted; the step and the forward program refuse it
                for refused in (lambda: bad.step(k, 8), lambda: bad.step(k, 8), bad.final_loss, bad.infer):
                    with pytest.raises(M.MsxError) as err:
                        refused()
                    assert err.value.status == M.BAD_INPUT and "labels" in str(err.value)
                with pytest.raises(M.MsxError):
                    bad.set_input("labels", y[:7])
                bad.set_input("labels", y)
                # The step plan's own inputs are another caller's: the run's batch is what its step reads.
                bad.step_plan.set_input("x", np.zeros((8, 12), dtype=np.float32))
                assert_bits_equal(bad.get_input("x", 96), (x + k).reshape(-1))
            good.step(k, 8); bad.step(k, 8)
            assert good.loss_of(k) == bad.loss_of(k)
    finally:
        good.destroy(); bad.destroy()


def test_kernels_that_start_early_give_the_same_bits(device):
    """MSX_FUSE bit 128: kernels of a captured step launched while the one before them ends. The same kernels on the same
    values: every loss, parameter and moment has the same bits with the bit on and off, in both precisions."""
    import json
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    results = []
    for mask in ("127", "255"):
        env = dict(os.environ, MSX_FUSE=mask, PYTHONPATH=os.pathsep.join([os.path.dirname(here), here, os.environ.get("PYTHONPATH", "")]))
        done = subprocess.run([sys.executable, os.path.join(here, "fuse_worker.py")], env=env, capture_output=True, text=True, timeout=600)
        assert done.returncode == 0, done.stderr[-2000:]
        results.append(json.loads(done.stdout.strip().splitlines()[-1]))
    for precision in ("f32", "bf16"):
        assert results[0][precision]["losses"] == results[1][precision]["losses"], precision
        assert results[0][precision]["state"] == results[1][precision]["state"], precision
