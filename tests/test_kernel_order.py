"""Synchronisation that no run can be relied on to miss, read from the kernels' source.

Shared memory of another block of a cluster may be written only after a cluster
barrier has shown that the block has started (CUDA programming guide,
distributed shared memory)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpir_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _bodies(src, head):
    """(name, body) of the functions whose declaration `head` (one group: the name) matches."""
    out = []
    for m in re.finditer(head, src):
        i = src.index("{", src.index(")", m.end()))
        depth, j = 0, i
        while True:
            depth += {"{": 1, "}": -1}.get(src[j], 0)
            j += 1
            if depth == 0:
                break
        out.append((m.group(1), src[i:j]))
    return out


def test_cluster_stores_follow_a_barrier():
    kernels = _bodies(_source("arnoldi.cu"), r"__global__[^;{]*?\b(k_gmres_\w+)\(")
    assert {k for k, _ in kernels} == {"k_gmres_begin", "k_gmres_first", "k_gmres_step", "k_gmres_end"}
    for name, body in kernels:
        first = min(m.start() for m in re.finditer(r"Reducer<|cluster_put\(|safe_norm\(", body))
        before = body[:first]
        assert re.search(r"cluster_sync\(\)|cluster_arrive\(\)[\s\S]*cluster_wait\(\)", before), name
