"""Distributed shared memory may be touched once every block of the cluster is
known to have started, and until none of them has ended: a kernel that maps
another block's shared memory passes a cluster barrier before the first such
access and another after the last."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "medyan_b200", "csrc")


def body_around(text, at):
    """The function body (top-level braces) that holds position at."""
    depth, start = 0, 0
    for m in re.finditer(r"[{}]", text):
        if m.group() == "{":
            depth += 1
            if depth == 1:
                start = m.end()
        else:
            depth -= 1
            if depth == 0 and start <= at < m.start():
                return text[start:m.start()]
    raise AssertionError("not in a function")


def test_cluster_barriers_enclose_distributed_shared_memory():
    kernels = 0
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        text = re.sub(r"^namespace \w* ?\{$", "", text, flags=re.M)  # so that functions are at depth one
        uses = [m.start() for m in re.finditer(r"map_shared_rank|mapa\.", text)]
        for at in uses:
            body = body_around(text, at)
            first, last = body.index(text[at:at + 5]), body.rindex(text[at:at + 5])
            sync = [m.start() for m in re.finditer(r"cluster\.sync\(\)|barrier\.cluster\.wait", body)]
            assert sync and sync[0] < first, f"{name}: no cluster barrier before the first access"
            assert sync[-1] > last, f"{name}: no cluster barrier after the last access"
            kernels += 1
    assert kernels > 0
