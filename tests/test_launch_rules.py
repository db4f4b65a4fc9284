"""Kernels that are launched while the one before still runs (launch.cuh) read
nothing that a kernel writes through the read-only path: the wait at their
beginning does not order such loads."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cpp-pt_gb300", "csrc")
# written by the host before a render's first launch
TABLES = {"DevBatchJob", "DevNNJob"}
LOOP_DATA = r"\b(PathIO|ShadowIO|PathBuffers|PathInput|WaveCounters|NNPathData|PPGVerts|NNMixture)\b"


def functions(text):
    """(head, body) of every function or struct with a body, by matching braces."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"^(?:__global__|__device__|struct)\b[^;{]*\{", text, re.M):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(0), text[m.end():i]


def read_only(code):
    return [t for t in re.findall(r"const\s+([\w ]+?)\s*\*\s*__restrict__", code) if t not in TABLES]


def test_no_read_only_loads_of_loop_buffers():
    kernels = helpers = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        for head, body in functions(open(os.path.join(CSRC, name)).read()):
            overlaps = head.startswith("__global__") and "after_previous()" in body
            if not overlaps and (head.startswith("__global__") or not re.search(LOOP_DATA, head)):
                continue
            kernels += overlaps
            helpers += not overlaps
            assert not read_only(head + body), (name, head)
    assert kernels >= 12 and helpers >= 4, (kernels, helpers)


def test_overlapping_launches_begin_with_the_wait():
    """Every kernel given to launch_after waits before anything else."""
    launched, waiting = set(), set()
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = open(os.path.join(CSRC, name)).read()
        launched |= set(re.findall(r"launch_after\((k_\w+)", text))
        for head, body in functions(text):
            if head.startswith("__global__") and body.lstrip().startswith("after_previous();"):
                waiting.add(re.search(r"\b(k_\w+)\(", head).group(1))
    assert launched and launched <= waiting, launched - waiting


def test_traversal_stacks_are_aligned():
    """Closest-hit stacks are read and written eight bytes at a time."""
    found = 0
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            for decl in re.findall(r"extern __shared__[^;]*s_stack\[\];", open(os.path.join(CSRC, name)).read()):
                found += 1
                assert "__align__(16)" in decl, (name, decl)
    assert found >= 6
