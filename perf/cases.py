"""The work a user of this backend has it do, as cases that can be timed and compared.

A training case is a stretch of a training run through the host loop of the C ABI: every step gets
its own host batch (`Training.set_input`), is submitted (`Training.step`), and its loss is read a
few steps behind (`Training.loss_of`); at the end of the stretch the run's state (parameters and
AdamW moments) is read back, as a program does that checkpoints or inspects the run between
stretches. The smallest run reads its loss at once instead, as an interactive program does. An
inference case stages a batch and reads the prediction and the loss (`Training.infer`). A held-out
case evaluates the declared batches of a split (`Training.heldout_evaluate`). All shapes are those
of the repository's configurations and tests or lie in the ranges around them.
"""
import ctypes
import math

import numpy as np
import torch

import modelspec_b200 as M
from modelspec_b200 import models, synthetic

# The run length the schedule is written for; a measured stretch is a piece of its beginning.
RUN_STEPS = 10_000_000
WARMUP_STEPS = 1000
# How many steps behind the last submitted one a loss is read (8 are kept in flight).
LAG = 4


def _bert(name, dtype, steps, batch, seq, layers, heads, head_dim, ffn, vocab, kind="train", padded=False):
    return {"name": name, "kind": kind, "model": "bert", "dtype": dtype, "steps": steps, "batch": batch, "seq": seq, "layers": layers,
            "heads": heads, "head_dim": head_dim, "ffn": ffn, "vocab": vocab, "padded": padded}


def listed():
    return [
        # The reference's smallest example (8 x 4 inputs, one weight, SGD), one step with its loss
        # read at once: latency of the host path, the upload, the launch and the read-back.
        {"name": "linear_regression", "kind": "train", "model": "linear_regression", "dtype": "f32", "steps": 1},
        # The MLP classifier configuration (64 x 784 -> 128 -> 10, SGD): a handful of small launches
        # per step.
        {"name": "mlp_classifier", "kind": "train", "model": "mlp", "dtype": "f32", "steps": 32, "batch": 64, "inputs": 784, "hidden": 128,
         "classes": 10},
        # The reference's transformer-block benchmark: two post-LN layers, 8 sequences, SGD, no
        # dropout.
        {"name": "transformer_block", "kind": "train", "model": "block", "dtype": "f32", "steps": 16, "batch": 8, "seq": 128, "layers": 2,
         "heads": 2, "head_dim": 64, "ffn": 512, "optimizer": "sgd", "dropout": 0.0},
        # BERT-tiny pre-training, the configuration the benchmark is quoted on, in f32 and in mixed
        # precision.
        _bert("bert_tiny_f32", "f32", 32, 32, 128, 2, 2, 64, 512, 30522),
        _bert("bert_tiny_bf16", "bf16", 32, 32, 128, 2, 2, 64, 512, 30522),
        # BERT-mini pre-training in f32.
        _bert("bert_mini_f32", "f32", 16, 32, 128, 4, 4, 64, 1024, 30522),
        # BERT-base-shaped pre-training, the largest configuration: mixed precision as it is meant to
        # be run, and f32.
        _bert("bert_base_bf16", "bf16", 16, 32, 512, 12, 12, 64, 3072, 30522),
        _bert("bert_base_f32", "f32", 4, 32, 512, 12, 12, 64, 3072, 30522),
        # Sizes that no tile divides: a few short padded sequences, odd widths, a small vocabulary.
        _bert("bert_ragged_f32", "f32", 16, 5, 77, 3, 3, 33, 250, 1009, padded=True),
        # The same in mixed precision (whose plans take widths and key counts of multiples of 8).
        _bert("bert_ragged_bf16", "bf16", 16, 11, 200, 3, 5, 40, 712, 5003, padded=True),
        # `infer`: the forward program on a few sequences, its whole [rows, vocabulary] prediction
        # read back.
        _bert("infer_bert_tiny", "f32", 1, 4, 128, 2, 2, 64, 512, 30522, kind="infer"),
        # `--eval-every`: four held-out batches through the prediction plan, reduced on the device.
        _bert("heldout_bert_tiny", "f32", 4, 32, 128, 2, 2, 64, 512, 30522, kind="heldout"),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v))) // step * step or step


# A drawn case stays below this many FLOP and bytes a pass: about a third of the largest listed one.
MOST_FLOP = 1.2e13
MOST_FLOP_BF16 = 6e13
MOST_BYTES = 3e10


def draw(rng):
    """A case of the same ranges: an MLP, an encoder block or a BERT-shaped model, trained, used for
    inference or evaluated, in f32 or (BERT) mixed precision."""
    while True:
        model = rng.choice(["mlp", "block", "bert", "bert", "bert", "bert"])
        if model == "mlp":
            case = {"kind": "train", "model": "mlp", "dtype": "f32", "steps": rng.choice([1, 8, 32]), "batch": _log(rng, 1, 4096),
                    "inputs": _log(rng, 4, 4096), "hidden": _log(rng, 4, 2048), "classes": _log(rng, 2, 2000)}
        else:
            half = model == "bert" and rng.random() < 0.5
            # Widths and lengths are multiples of 8 or 16 more often than not.
            by = rng.choice([8, 8, 16]) if half else rng.choice([1, 8, 8, 16])
            case = {"kind": "train", "model": model, "dtype": "bf16" if half else "f32", "steps": rng.choice([2, 8, 16]),
                    "batch": _log(rng, 1, 64), "seq": _log(rng, 16, 512, by), "layers": rng.randint(1, 12), "heads": rng.randint(1, 12),
                    "head_dim": _log(rng, 16, 64, by), "ffn": _log(rng, 32, 3072, by)}
            if model == "block":
                case.update(optimizer=rng.choice(["sgd", "adamw"]), dropout=rng.choice([0.0, 0.1]))
            else:
                case.update(kind=rng.choice(["train", "train", "train", "infer", "heldout"]), vocab=_log(rng, 200, 50000),
                            padded=rng.random() < 0.5)
                if case["kind"] == "infer":
                    case["steps"] = 1
        w = work(case)
        prediction = case["kind"] == "infer" and 4 * case["batch"] * case["seq"] * case["vocab"]
        if w["flops"] <= (MOST_FLOP_BF16 if case["dtype"] == "bf16" else MOST_FLOP) and w["bytes"] <= MOST_BYTES and prediction <= 2.5e8:
            return case


# ---- sizes ---------------------------------------------------------------------------------------


def _masked(case):
    return models.default_masked_rows(case["batch"] * case["seq"])


def _hidden(case):
    return case["heads"] * case["head_dim"]


def _parameters(case):
    """How many parameter elements the case's model holds."""
    if case["model"] == "linear_regression":
        return 4
    if case["model"] == "mlp":
        return case["inputs"] * case["hidden"] + case["hidden"] + case["hidden"] * case["classes"] + case["classes"]
    h, f = _hidden(case), case["ffn"]
    layers = case["layers"] * (4 * h * h + 4 * h + 2 * h * f + f + h + 4 * h)
    if case["model"] == "block":
        return layers
    return layers + case["vocab"] * h + case["seq"] * h + 2 * h + h * h + 3 * h + case["vocab"]


def _forward_flop(case, head_rows):
    if case["model"] == "linear_regression":
        return 2 * 8 * 4
    if case["model"] == "mlp":
        return 2 * case["batch"] * (case["inputs"] * case["hidden"] + case["hidden"] * case["classes"])
    h, rows = _hidden(case), case["batch"] * case["seq"]
    flop = case["layers"] * (8 * rows * h * h + 4 * rows * h * case["ffn"] + 4 * rows * case["seq"] * h)
    if case["model"] == "bert":
        flop += 2 * head_rows * h * (h + case["vocab"])
    return flop


def _batch_bytes(case):
    if case["model"] == "linear_regression":
        return 4 * (8 * 4 + 8)
    if case["model"] == "mlp":
        return 4 * (case["batch"] * (case["inputs"] + 2))
    rows = case["batch"] * case["seq"]
    return 4 * rows * (5 if case["model"] == "bert" else 2 * _hidden(case) + 1)


def work(case):
    """One pass: the products of its steps, and its inputs, its parameters and their state read and
    written once a step, and what is read back."""
    p, steps = _parameters(case), case["steps"]
    if case["kind"] == "train":
        words = 3 if _adamw(case) else 1
        head_rows = _masked(case) if case["model"] == "bert" else 0
        # Forward, and two products of the same size for each one backward.
        flop = 3 * _forward_flop(case, head_rows)
        return {"flops": steps * flop, "bytes": steps * (8 * words * p + _batch_bytes(case) + 4) + 4 * words * p}
    rows = case["batch"] * case["seq"]
    out = 4 * rows * case["vocab"] if case["kind"] == "infer" else 0
    return {"flops": steps * _forward_flop(case, rows), "bytes": 4 * p + steps * (_batch_bytes(case) + out)}


def tolerance(case):
    """f32 plans multiply in split TF32 with f32 sums; a training stretch carries the rounding of
    one step into the next ones (two plans of this repository, exact and split products, differ by
    up to 2e-5 in the moments). A mixed-precision plan stores activations as bf16 (8 significant
    bits): its gradients move by up to 1e-2 as a whole and single elements by their own size when
    one rounding falls the other way."""
    if case["dtype"] == "bf16":
        return {"rel": 2e-2, "max": 0.99}
    return {"rel": 1e-4} if case["kind"] == "train" else {"rel": 2e-5}


# ---- models and batches --------------------------------------------------------------------------


def _adamw(case):
    return case["model"] == "bert" or case.get("optimizer") == "adamw"


def _source(case, seed):
    if case["model"] == "linear_regression":
        return models.linear_regression(steps=RUN_STEPS, seed=seed), 0
    if case["model"] == "mlp":
        return models.mlp_classifier(batch=case["batch"], inputs=case["inputs"], hidden=case["hidden"], classes=case["classes"],
                                     steps=RUN_STEPS, seed=seed), 0
    if case["model"] == "block":
        more = dict(lr=1e-3, weight_decay=0.01, eps=1e-6, warmup_steps=WARMUP_STEPS) if case["optimizer"] == "adamw" else dict(lr=0.01)
        return models.transformer_block(batch=case["batch"], seq=case["seq"], hidden=_hidden(case), heads=case["heads"], ffn=case["ffn"],
                                        layers=case["layers"], dropout=case["dropout"], optimizer=case["optimizer"], steps=RUN_STEPS,
                                        seed=seed, **more), 0
    source = models.bert(layers=case["layers"], hidden=_hidden(case), heads=case["heads"], ffn=case["ffn"], vocab=case["vocab"],
                         seq=case["seq"], batch=case["batch"], warmup_steps=WARMUP_STEPS, steps=RUN_STEPS, seed=seed)
    return source, _masked(case)


def _batch(case, seed, k):
    """Batch `k` of the run: what the declared inputs and targets hold."""
    rng = np.random.default_rng([seed, k])
    if case["model"] == "linear_regression":
        x = rng.standard_normal((8, 4), dtype=np.float32)
        return {"x": x, "y": x @ np.array([[1.0], [-2.0], [0.5], [3.0]], dtype=np.float32)}
    if case["model"] == "mlp":
        return {"x": rng.random((case["batch"], case["inputs"]), dtype=np.float32),
                "labels": rng.integers(0, case["classes"], case["batch"], dtype=np.int32), "weights": np.ones(case["batch"], dtype=np.float32)}
    rows = case["batch"] * case["seq"]
    if case["model"] == "block":
        return {"x": rng.standard_normal((rows, _hidden(case)), dtype=np.float32), "key_mask": np.ones(rows, dtype=np.float32),
                "y": rng.standard_normal((rows, _hidden(case)), dtype=np.float32)}
    # Zipf token ids, 15 % of the positions masked as the reference masks them.
    batch = synthetic.mlm_batch(k, seed=seed, batch=case["batch"], seq=case["seq"], vocab=case["vocab"])
    if case["padded"]:
        # Sequences of half to full length; what lies behind a sequence's end is neither attended to
        # nor predicted.
        length = rng.integers((case["seq"] + 1) // 2, case["seq"] + 1, case["batch"])
        inside = (np.arange(case["seq"])[None, :] < length[:, None]).reshape(-1)
        batch["key_mask"] = inside.astype(np.float32)
        batch["weights"] = batch["weights"] * batch["key_mask"]
        batch["ids"] = np.where(inside, batch["ids"], 0).astype(np.int32)
    return batch


# ---- the cases -----------------------------------------------------------------------------------

_device = None


def _open():
    global _device
    if _device is None:
        _device = M.Device(0)
    return _device


class Run:
    """What a program keeps between its calls: the run, its next batches, and the pinned buffers
    its state is read back into."""

    def __init__(self, case, seed):
        source, masked_rows = _source(case, seed)
        self.case = case
        self.training = M.Training(_open(), source, masked_rows, M.PLAN_BF16 if case["dtype"] == "bf16" else M.PLAN_DEFAULT)
        self.batches = [_batch(case, seed, k) for k in range(case["steps"])]
        self.at = 0
        if case["kind"] == "train":
            self.sizes = [nbytes for _, nbytes in self.training.step_plan.params()]
            self.state = [torch.empty(sum(self.sizes) // 4, dtype=torch.float32, pin_memory=True) for _ in range(3 if _adamw(case) else 1)]
        if case["kind"] == "heldout":
            self.training.heldout_begin(case["steps"], "labels", "weights")
            for b, batch in enumerate(self.batches):
                for name, value in batch.items():
                    self.training.heldout_set(b, name, value)

    def __del__(self):
        training = getattr(self, "training", None)
        if training is not None:
            training.destroy()

    def train(self):
        run, steps = self.training, self.case["steps"]
        losses = np.empty(steps, dtype=np.float32)
        for k, batch in enumerate(self.batches):
            for name, value in batch.items():
                run.set_input(name, value)
            run.step(self.at + k, RUN_STEPS)
            if k >= LAG:
                losses[k - LAG] = run.loss_of(self.at + k - LAG)
        for k in range(max(0, steps - LAG), steps):
            losses[k] = run.loss_of(self.at + k)
        self.at += steps
        return [losses] + self.read_state()

    def read_state(self):
        """The parameters, and the AdamW moments, in parameter order."""
        plan, check = self.training.step_plan.h, self.training.step_plan.device.check
        at = 0
        for i, nbytes in enumerate(self.sizes):
            for which, buffer in zip(("p", b"m", b"v"), self.state):
                to = ctypes.c_void_p(buffer.data_ptr() + at)
                if which == "p":
                    check(M.lib().msx_param_download(plan, i, to, nbytes))
                else:
                    check(M.lib().msx_moment_download(plan, i, which, to, nbytes))
            at += nbytes
        return self.state

    def infer(self):
        for name, value in self.batches[0].items():
            self.training.set_input(name, value)
        prediction, loss = self.training.infer()
        return [prediction, np.array([loss], dtype=np.float32)]

    def evaluate(self):
        return np.array(self.training.heldout_evaluate(), dtype=np.float32)


def prepare(case, seed):
    return Run(case, seed)


def run(state):
    kind = state.case["kind"]
    return state.train() if kind == "train" else state.infer() if kind == "infer" else state.evaluate()
