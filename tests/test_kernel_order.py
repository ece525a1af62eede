"""In a captured step a kernel may be launched while the one before it still runs (common.cuh, chain_kernels): every kernel
that a step can hold has to wait for its producers before it touches memory."""
import glob
import os
import re

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "modelspec_b200", "csrc", "cuda")
# Never in a graph whose edges are changed: an entry point of its own, and the exchange between ranks.
OUTSIDE = {"noalloc.cu", "peer_reduce.cu"}
WAITS = ("after_producers()", "wait_for_producers()")


def kernels():
    for path in sorted(glob.glob(os.path.join(CUDA, "*.cu"))):
        if os.path.basename(path) in OUTSIDE:
            continue
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for at in re.finditer(r"__global__", text):
            start, depth = text.index("{", at.end()), 0
            head = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text[at.end():start])
            name = re.search(r"(\w+)\s*\(", head).group(1)
            for end in range(start, len(text)):
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                if depth == 0:
                    break
            yield os.path.basename(path), name, text[start + 1:end], text


# Kernels that set up barriers and tensor memory first, and then wait.
SET_UP_FIRST = {"matmul_tc_kernel", "tf32_kernel", "bf16_kernel", "attention_forward_kernel", "attention_backward_kernel",
                "attention_backward_whole_kernel", "attention_f32_forward_kernel", "attention_f32_backward_kernel"}


def test_every_kernel_of_a_step_waits_for_its_producers():
    names = set()
    for path, name, body, text in kernels():
        names.add(name)
        if name not in SET_UP_FIRST:
            assert body.strip().startswith("after_producers();"), "%s: %s touches memory before it waits" % (path, name)
        elif not any(w in body for w in WAITS):
            # In the function that does the whole work of a block, or sets it up.
            assert re.search(r"\b(begin|backward_rows|backward_keys|backward_queries)\s*[<(]", body) and any(w in text for w in WAITS), "%s: %s never waits" % (path, name)
    assert SET_UP_FIRST <= names and len(names) > 50
