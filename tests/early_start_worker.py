"""Child process of test_gpu_early_starts.py: trains, evaluates and infers at sizes whose kernels take several waves, under the MSX_FUSE mask of
its environment (read once per process), and prints the bits of every result. No loss is read between the steps."""
import hashlib
import json
import sys

import numpy as np

import modelspec_b200 as M
from modelspec_b200 import models, synthetic

BERT = {
    # name: layers, heads, head width, ffn, vocabulary, batch, sequence, steps, held-out batches
    "tiny": (2, 2, 64, 512, 30522, 32, 128, 5, 2),
    "mini": (4, 4, 64, 1024, 30522, 32, 128, 3, 0),
    "wide": (1, 12, 64, 3072, 8000, 16, 256, 3, 0),  # (bf16: the gradients of attention by whole heads)
    "long": (2, 2, 48, 200, 3000, 3, 512, 4, 0),     # (bf16: by blocks of queries and of keys, of several tiles)
}
RAGGED = {"f32": (3, 3, 33, 250, 1009, 5, 77, 5, 1), "bf16": (3, 5, 40, 712, 5003, 11, 200, 5, 1)}


def digest(*values):
    h = hashlib.sha256()
    for v in values:
        h.update(v if isinstance(v, bytes) else np.ascontiguousarray(v).tobytes())
    return h.hexdigest()


def bert(device, flags, layers, heads, width, ffn, vocab, batch, seq, steps, heldout):
    hidden = heads * width
    source = models.bert(layers=layers, hidden=hidden, heads=heads, ffn=ffn, vocab=vocab, seq=seq, batch=batch, warmup_steps=1, steps=steps)
    run = M.Training(device, source, models.default_masked_rows(batch * seq), flags)
    try:
        batches = [synthetic.mlm_batch(k, batch=batch, seq=seq, vocab=vocab) for k in range(steps)]
        if heldout:
            run.heldout_begin(heldout, "labels", "weights")
            for b in range(heldout):
                for name, value in batches[b].items():
                    run.heldout_set(b, name, value)
        for k, values in enumerate(batches):
            for name, value in values.items():
                run.set_input(name, value)
            run.step(k, steps)
        out = {"losses": [int(np.float32(run.loss_of(k)).view(np.uint32)) for k in range(steps)]}
        ckpt = run.checkpoint(steps)
        out["state"] = digest(ckpt.encode())
        ckpt.destroy()
        if heldout:
            out["heldout"] = digest(np.array(run.heldout_evaluate(), dtype=np.float32))
        if batch * seq * vocab < 4e6:
            prediction, loss = run.infer()
            out["infer"] = digest(prediction, np.float32(loss))
        return out
    finally:
        run.destroy()


def plain(device, source, batches):
    run = M.Training(device, source)
    try:
        for k, values in enumerate(batches):
            for name, value in values.items():
                run.set_input(name, value)
            run.step(k, len(batches))
        losses = [int(np.float32(run.loss_of(k)).view(np.uint32)) for k in range(len(batches))]
        return {"losses": losses, "state": digest(*(run.step_plan.param_download(i) for i in range(len(run.step_plan.params()))))}
    finally:
        run.destroy()


def main():
    device = M.Device(0)
    out = {}
    for precision, flags in (("f32", M.PLAN_DEFAULT), ("bf16", M.PLAN_BF16)):
        for name, shape in dict(BERT, ragged=RAGGED[precision]).items():
            out["%s %s" % (name, precision)] = bert(device, flags, *shape)
    r = np.random.default_rng(0)
    out["mlp"] = plain(device, models.mlp_classifier(batch=64, inputs=784, hidden=128, classes=10, steps=7),
                       [{"x": r.random((64, 784), dtype=np.float32), "labels": r.integers(0, 10, 64, dtype=np.int32), "weights": np.ones(64, dtype=np.float32)}
                        for _ in range(7)])
    rows, hidden = 8 * 128, 128
    out["block"] = plain(device, models.transformer_block(batch=8, seq=128, hidden=hidden, heads=2, ffn=512, layers=2, dropout=0.0, optimizer="sgd", steps=5, lr=0.01),
                         [{"x": r.standard_normal((rows, hidden), dtype=np.float32), "key_mask": np.ones(rows, dtype=np.float32),
                           "y": r.standard_normal((rows, hidden), dtype=np.float32)} for _ in range(5)])
    print(json.dumps(out))


if __name__ == "__main__":
    sys.exit(main())
