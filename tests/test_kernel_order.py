"""Synchronisation that no run can be relied on to miss, read from the kernels' source.

Shared memory of another block of a cluster may be written only after a cluster
barrier has shown that the block has started (CUDA programming guide,
distributed shared memory).  Bulk copies write shared memory through the async
proxy: ordinary stores to the same bytes come before them only with a proxy
fence by the storing threads (PTX ISA, async proxy)."""
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


def test_bulk_copies_follow_a_proxy_fence():
    """The several-vector solves store vectors and partial sums inside the area of the
    inverse blocks; the single-vector ones keep theirs behind it (then no fence is needed)."""
    (_, loop), = _bodies(_source("flow_dev.cuh"), r"\b(flow_loop)\(")
    body = loop[loop.index("work("):]
    assert re.search(r"if \(kStores\) asm volatile\(\"fence\.proxy\.async\.shared::cta;\"[^;]*;[^;]*"
                     r"__syncthreads\(\)", body)
    for name, head, kinds in (("solve_multi.cu", r"\b(k_(?:fwd|bwd)_flow_m)\(const", {"true"}),
                              ("solve.cu", r"\b(k_(?:fwd|bwd)_flow)\(const", {"false"})):
        kernels = _bodies(_source(name), head)
        assert len(kernels) == 2
        assert {re.search(r"flow_loop<(\w+)>", b).group(1) for _, b in kernels} == kinds
    single = _source("solve.cu")
    stored = re.findall(r"\*\s*(\w+)\s*=\s*sm(\s*\+\s*kFlowInvSmem)?", single)
    assert stored and all(at or v == "inv" for v, at in stored)
    assert not re.search(r"\b(?:inv|blk|M)\[[^\]]*\]\s*[-+]?=[^=]", single[:single.index("k_flow_invert(")])
