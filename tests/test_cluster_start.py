"""The cluster rrLU writes to its peers' shared memory only after a cluster barrier
that every CTA passes once it has started.  A missing wait shows no wrong value on
most runs, so the order is checked in the source."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _body(text, head):
    """The function body that follows `head`, comments removed."""
    text = re.sub(r"//[^\n]*", "", text)
    start = text.index("{", text.index(")", text.index(head)))
    depth = 0
    for pos in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[pos], 0)
        if depth == 0:
            return text[start:pos]
    raise AssertionError(f"unbalanced braces after {head}")


def test_cluster_barrier_before_the_first_exchange():
    with open(os.path.join(ROOT, "tensorcrossinterpolation.jl_gb300", "csrc", "step_kernel.cu")) as fh:
        text = fh.read()
    body = _body(text, "ClusterResult cluster_rrlu(const ClusterJob& P")
    first = min(body.index("cluster_exchange("), body.index("map_shared_rank"))
    before = body[:first]
    loop = before.index("while (P.kmax > 0)")
    arrive, wait = before.index("barrier.cluster.arrive"), before.index("barrier.cluster.wait")
    assert arrive < wait < loop  # outside the loop: passed by every launch
    # nothing reaches a peer's shared memory but through that function and its helpers
    for kernel in ("rrlu_cluster_task_kernel(const tci_task T", "rrlu_noalloc_cluster_kernel(const double*"):
        assert "map_shared_rank" not in _body(text, kernel)
        assert "cluster_rrlu<" in _body(text, kernel)
