"""Blocks of a cluster write to each other's shared memory only once all of
them have started: in every kernel of many.cu the sums that do so come after
a cluster barrier.  Read from the source, since a store to a block that has
not started is nothing a test may provoke on a GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ogs5_gb300", "csrc")


def _body(text, start):
    """The braces' content after position start."""
    i = text.index("{", start)
    depth = 0
    for k in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[i + 1:k]
    raise AssertionError("unbalanced braces")


def test_remote_stores_follow_a_cluster_barrier():
    with open(os.path.join(CSRC, "many.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    kernels = [m for m in re.finditer(r"__global__ void [^;{]*?(k_\w+)\(", text)]
    assert {m.group(1) for m in kernels} >= {"k_cg_many", "k_bi_many"}
    enter = re.search(r"void enter\(\)", text)
    assert enter and re.search(r"if \(CLUSTER\) many_cluster_sync\(\);", _body(text, enter.start()))
    # the only remote stores are those of sum()
    assert len(re.findall(r"cluster_store\(", text)) == 2  # its definition and the call in sum()
    assert "cluster_store(" in _body(text, text.index("bool sum("))
    for m in kernels:
        body = _body(text, m.end())
        first = re.search(r"sync\.(\w+)\(", body)
        assert first and first.group(1) == "enter", m.group(1)
        # nothing else may leave the kernel between its start and the barrier but `done`
        assert body[:first.start()].count("return") == 1 and "if (st->done) return;" in body[:first.start()]
