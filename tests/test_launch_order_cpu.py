"""Overlapping launches: a kernel releases its successor only behind its own wait for its predecessor, so at most two kernels of a stream are in flight and a
kernel that holds tensor memory, shared memory or SMs of a cluster while it waits can only wait for one that already has all it needs."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm-inference-engine_b200", "csrc")


def kernels(text):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__", text):
        head = re.compile(r"(\w+_kernel)\s*\(").search(text, m.end())
        at = depth = head.end() - 1
        depth = 0
        while True:  # end of the parameter list
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
            if depth == 0:
                break
        rest = text[at:].lstrip()
        if not rest.startswith("{"):
            continue  # a declaration
        start = end = text.index("{", at)
        depth = 0
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield head.group(1), text[start:end]


def test_successors_are_released_behind_the_wait():
    seen = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for name, body in kernels(text):
            release = body.find("pdl_launch_dependents()")
            if release >= 0:
                wait = body.find("pdl_wait()")
                seen[name] = 0 <= wait < release
    assert len(seen) >= 8 and {"norm_kernel", "gemm_tc_kernel", "gemm_tc_pair_kernel", "gemv_rs_kernel", "topk_stage1_kernel"} <= set(seen), seen
    assert all(seen.values()), [n for n, ok in seen.items() if not ok]
