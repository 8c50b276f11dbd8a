"""Kernels that write another block's shared memory wait until every block of the cluster has
begun.  CUDA leaves an earlier access undefined, and one that goes wrong loses a box without an
error, so the order is checked in the source: nothing on a GPU would show it reliably."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cccollisions_b200", "csrc")


def _kernels():
    """(name, body without comments) of every kernel of the sources."""
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\([^{;]*\)\s*\{", text):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield m.group(1), text[m.end():end]


def test_blocks_of_a_cluster_have_begun_before_their_shared_memory_is_used():
    found = 0
    for name, body in _kernels():
        if "map_shared_rank" not in body:
            continue
        found += 1
        # ahead of the mapping, and in the kernel's own scope: reached by every block
        before = body[:body.index("map_shared_rank")]
        assert "cluster.sync();" in before, name
        head = before[:before.index("cluster.sync();")]
        assert head.count("{") == head.count("}") and "return" not in head, name
    assert found == 1
