"""A run's batch is the run's until one of its steps has checked it, however it waits (inputs of 4 KB and more lie in the slot of
the next step already): what else runs the step plan reads what that plan was last given, a refused batch included."""
import numpy as np
import pytest

import modelspec_b200 as M
import packed_dir
from helpers import assert_bits_equal
from modelspec_b200 import models, synthetic

pytestmark = pytest.mark.gpu

# 1,024 rows: ids, labels, weights and the key mask have 4,096 bytes each.
BATCH, SEQ, VOCAB, STEPS = 8, 128, 304, 40
SOURCE = models.bert(name="BertTiny", hidden=32, heads=2, ffn=64, vocab=VOCAB, seq=SEQ, batch=BATCH, warmup_steps=2, steps=STEPS)


def batch_of(k):
    return synthetic.mlm_batch(k, vocab=VOCAB, seq=SEQ, batch=BATCH)


def feed(run, k):
    for name, value in batch_of(k).items():
        run.set_input(name, value)


def state(run):
    ckpt = run.checkpoint(STEPS)
    try:
        return ckpt.encode()
    finally:
        ckpt.destroy()


@pytest.fixture
def pair(device):
    runs = [M.Training(device, SOURCE, 192) for _ in range(2)]
    yield runs
    for run in runs:
        run.destroy()


@pytest.mark.parametrize("how", ["run", "profile_step", "profile_report"])
@pytest.mark.parametrize("before", [1, 7, 8, 9])  # (the slots are eight)
def test_a_step_of_the_plan_alone_runs_the_batch_it_has(pair, how, before):
    early, late = pair
    for k in range(before):
        for run in pair:
            feed(run, k); run.step(k, STEPS)
        assert early.loss_of(k) == late.loss_of(k)
    for repeat in range(2):
        feed(early, before)  # the next batch, in front of what runs the last one again
        for run in pair:
            getattr(run.step_plan, how)()
        assert early.step_plan.loss() == late.step_plan.loss()
    for name, value in batch_of(before).items():
        assert_bits_equal(early.get_input(name, value.size, value.dtype), value.reshape(-1))
    feed(late, before)
    for run in pair:
        run.step(before, STEPS)
    assert early.loss() == late.loss()
    assert state(early) == state(late)


def test_a_refused_batch_reaches_no_step(pair):
    bad, little = pair
    for k in range(4):
        batch = batch_of(k)
        half = batch["key_mask"].copy().reshape(-1); half[5] = 0.5  # neither 0 nor 1
        feed(bad, k)
        if k == 0:
            feed(little, k)
        # The plan has the inputs whose names come before the refused one's, and no other: `little` has set no other.
        for run in pair:
            run.set_input("ids", batch["ids"]); run.set_input("key_mask", half)
            for _ in range(2):
                with pytest.raises(M.MsxError) as err:
                    run.step(k, STEPS)
                assert err.value.status == M.BAD_INPUT and "key_mask" in str(err.value)
            assert_bits_equal(run.get_input("key_mask", half.size), half)
            if k:
                run.step_plan.run()
        if k:
            assert bad.step_plan.loss() == little.step_plan.loss()
        bad.set_input("key_mask", batch["key_mask"])
        feed(little, k)
        for run in pair:
            run.step(k, STEPS)
        assert bad.loss() == little.loss()
    assert state(bad) == state(little)


def test_another_caller_s_values_are_the_plan_s_and_the_run_s_batch_the_run_s(pair):
    """`msx_set_input` over what the run has staged, and over what its last step has accepted."""
    mine, other = pair
    for k in range(4):
        batch, strange = batch_of(k), batch_of(100 + k)
        strange["key_mask"] = np.ascontiguousarray(np.roll(np.tril(np.ones((SEQ, SEQ), dtype=np.float32)), k, 0)[:BATCH]).reshape(-1)
        for run in pair:
            if k != 2:
                feed(run, k)
        for run, names in ((mine, ("ids", "key_mask")), (other, ())):
            for name in names:
                run.step_plan.set_input(name, strange[name])
                expected = (batch if k != 2 else batch_of(1))[name].reshape(-1)
                assert_bits_equal(run.get_input(name, expected.size, expected.dtype), expected)
        for run in pair:
            run.step(k, STEPS)
        assert mine.loss_of(k) == other.loss_of(k)
    # And as the plan's they are what it runs.
    strange = batch_of(200)
    feed(mine, 50)
    for run in pair:
        run.step_plan.set_input("ids", strange["ids"])
        run.step_plan.run()
    assert mine.step_plan.loss() == other.step_plan.loss()
    assert state(mine) == state(other)


def test_steps_submitted_without_a_wait_read_the_batches_they_were_given(device):
    """More steps than slots in flight: what is set while no slot is free waits beside them."""
    source = models.bert(name="BertTiny", hidden=256, heads=4, ffn=512, vocab=8000, seq=SEQ, batch=32, warmup_steps=2, steps=STEPS)
    losses = []
    for lag in (0, 7):
        run = M.Training(device, source, models.default_masked_rows(32 * SEQ))
        try:
            mine = []
            for k in range(STEPS):
                for name, value in synthetic.mlm_batch(k, vocab=8000, seq=SEQ, batch=32).items():
                    run.set_input(name, value)
                run.step(k, STEPS)
                if k >= lag:
                    mine.append(run.loss_of(k - lag))
            mine += [run.loss_of(k) for k in range(STEPS - lag, STEPS)]
            losses.append(mine)
        finally:
            run.destroy()
    assert losses[0] == losses[1] and len(losses[0]) == STEPS


def test_a_rewind_and_the_feeds_replace_what_was_set(pair, device, tmp_path):
    straight, run = pair
    for k in range(6):
        feed(straight, k); straight.step(k, STEPS)
    expected = state(straight)
    run.set_replay_window(4)
    for k in range(8):
        feed(run, k); run.step(k, STEPS)
    feed(run, 30)
    run.rewind(5)
    assert state(run) == expected
    for k in (6, 7):
        for r in pair:
            feed(r, k); r.step(k, STEPS)
        assert straight.loss() == run.loss()
    # A packed feed over a staged batch draws what it draws over none.
    r = np.random.default_rng(1)
    train, heldout = (r.integers(110, VOCAB, size=40 * SEQ).astype(np.int32) for _ in range(2))
    packed_dir.write(str(tmp_path / "packed"), train, heldout, SEQ, VOCAB)
    packs = [M.Packed(str(tmp_path / "packed")) for _ in pair]
    for one, pack in zip(pair, packs):
        one.bind_packed(pack)
    for k in (8, 9):
        feed(run, 60 + k)
        for one in pair:
            one.feed_packed(k); one.step(k, STEPS)
        assert straight.loss() == run.loss()
    # And a dense one.
    batches = [batch_of(k) for k in range(4)]
    for name in batches[0]:
        files = np.concatenate([np.asarray(b[name]).reshape(-1) for b in batches])
        files.tofile(str(tmp_path / (name + (".f32" if files.dtype == np.float32 else ".i32"))))
    for one in pair:
        one.bind_dense(str(tmp_path))
    for k in (10, 11):
        feed(run, 70 + k)
        for one in pair:
            one.feed_dense(k); one.step(k, STEPS)
        assert straight.loss() == run.loss()
    assert state(straight) == state(run)
    for pack in packs:
        pack.close()
