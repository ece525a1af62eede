"""In a captured step a kernel may be launched while the one before it still runs (common.cuh, chain_kernels): every kernel
that a step can hold has to wait for its producers before it touches memory, and to read with ordinary loads, which the compiler
and the device keep behind that wait. By the source's text: what the compiler makes of it is compared on the device
(test_gpu_early_starts.py)."""
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


# What reads or writes global memory, or starts a copy that does.
TOUCHES = re.compile(r"\b(load[148]|load2|load_row|load_global|load_settled|settled|store[1248]|fetch|fetch4|fetch_row|put_row|tma_load|load_tile|atomicAdd|statistics|"
                     r"keys_that_count)\s*[<(]")


def without_lambdas(text):
    """The statements of a body, without those of the functions it defines for later."""
    while True:
        at = re.search(r"auto \w+ = \[[^\]]*\]\s*\([^{};]*\)[^{};]*\{", text)
        if not at:
            return text
        depth, end = 1, at.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        text = text[:at.start()] + text[end:]


def test_every_kernel_of_a_step_waits_for_its_producers():
    names = set()
    for path, name, body, text in kernels():
        names.add(name)
        if name not in SET_UP_FIRST:
            assert body.strip().startswith("after_producers();"), "%s: %s touches memory before it waits" % (path, name)
        elif not any(w in body for w in WAITS):
            # In the function that does the whole work of a block, or sets it up.
            assert re.search(r"\b(begin|backward_rows|backward_keys|backward_queries)\s*[<(]", body) and any(w in text for w in WAITS), "%s: %s never waits" % (path, name)
            ahead = without_lambdas(body)
            ahead = ahead[: re.search(r"\b(begin|backward_rows|backward_keys|backward_queries)\s*[<(]", ahead).start()]
            assert not TOUCHES.search(ahead), "%s: %s touches memory before it waits" % (path, name)
        else:
            ahead = without_lambdas(body)
            ahead = ahead[: min(ahead.index(w) for w in WAITS if w in ahead)]
            assert not TOUCHES.search(ahead), "%s: %s touches memory before it waits" % (path, name)
    assert SET_UP_FIRST <= names and len(names) > 50


def test_the_functions_that_wait_within_a_kernel_touch_nothing_before():
    seen = set()
    for path in ("attention_f32.cu", "attention_fused.cu"):
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CUDA, path)).read())
        for at in re.finditer(r"__device__ __forceinline__ \w+ (begin|backward_rows|backward_keys|backward_queries)\(([^)]*)\) \{", text):
            depth, end = 1, at.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            body = without_lambdas(text[at.end():end])
            seen.add(at.group(1))
            waits = [body.index(w) for w in WAITS + ("begin(ctl)",) if w in body]
            assert waits and not TOUCHES.search(body[: min(waits)]), "%s: %s touches memory before it waits" % (path, at.group(1))
            assert "__restrict__" not in at.group(2)
    assert seen == {"begin", "backward_rows", "backward_keys", "backward_queries"}


def test_kernels_of_a_step_read_with_ordinary_loads():
    """What a kernel's `const __restrict__` parameter points to, and what __ldg and ld.global.nc read, nobody may write while the kernel
    runs: that does not hold of a kernel that starts while its producer runs, and the compiler may move such loads ahead of the wait."""
    for path in sorted(glob.glob(os.path.join(CUDA, "*.cu")) + glob.glob(os.path.join(CUDA, "*.cuh"))):
        if os.path.basename(path) in OUTSIDE:
            continue
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for found in ("__ldg", "ld.global.nc", "ld.global.L1", "__ldca", "__ldcg(reinterpret"):
            assert found not in text, (path, found)
        for at in re.finditer(r"__global__", text):
            assert "__restrict__" not in text[at.start():text.index("{", at.end())], (path, text[at.start():at.start() + 120])
