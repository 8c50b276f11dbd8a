"""A tree that leads back to a node is refused, and no later than by one thread a query."""
import ctypes

import numpy as np
import pytest
import torch


def _query(lib, boxes, tree, x0, x1, mask, binary_nodes):
    """(status, milliseconds) of a masked continuous query, with all of its scratch or with just
    enough for the binary nodes, which one thread a query walks."""
    from cccollisions_b200 import _native as N
    B, F = x0.shape[:2]
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    size = lib.ccc_workspace_size(N.OP_CONTINUOUS, B, F, 4)
    if binary_nodes:
        size -= (64 * B * F // 256 - 1) * 256
    ws = torch.empty(size, dtype=torch.uint8, device=x0.device)
    rows = torch.full((B, F, 3), -1, dtype=torch.int64, device=x0.device)
    times = torch.full((B, F, 1), -1, dtype=x0.dtype, device=x0.device)
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    a.record()
    assert lib.ccc_find_collisions_continuous(int(x0.dtype == torch.float64), p(boxes), p(tree), p(x0), p(x1), p(mask),
                                              B, F, 4, 1, p(rows), p(times), p(ws), size,
                                              torch.cuda.current_stream().cuda_stream) == 0
    b.record()
    out = (ctypes.c_int32 * 4)()
    assert lib.ccc_read_counters(p(ws), out, torch.cuda.current_stream().cuda_stream) == 0
    return out[0], a.elapsed_time(b)


@pytest.mark.gpu
@pytest.mark.parametrize("turning", ["every query", "one of a group"])
def test_a_circle_ends(cuda, native_lib, turning):
    import cccollisions_b200 as C
    from cccollisions_b200 import _native as N
    F = 20000
    g = torch.Generator(device=cuda).manual_seed(3)
    x0 = torch.rand((1, F, 3, 3), generator=g, device=cuda) * 0.01 + torch.rand((1, F, 1, 3), generator=g, device=cuda)
    x1 = x0.clone()
    boxes, tree = C.bvh_motion(x0, x1)
    # the root's left child leads to leaf 0 and back to itself
    node = int(tree[0, 0, 1])
    tree[0, node, 1], tree[0, node, 2] = F - 1, node
    # the queries that meet that node go round it: all of them, or those with a box that large
    if turning == "every query":
        boxes[0, node] = torch.tensor([-1.0, -1, -1, 2, 2, 2], device=cuda)
    else:
        boxes[0, node] = torch.tensor([5.0, 5, 5, 6, 6, 6], device=cuda)
        boxes[0, F - 1 + 15::32] = torch.tensor([-1.0, -1, -1, 6, 6, 6], device=cuda)
    mask = torch.ones((1, F), dtype=torch.uint8, device=cuda)
    times = {}
    for binary_nodes in (True, False):
        runs = [_query(native_lib, boxes, tree, x0, x1, mask, binary_nodes) for _ in range(4)]
        assert all(status & N.CCC_ST_MALFORMED_TREE for status, _ in runs)
        times[binary_nodes] = float(np.median([ms for _, ms in runs[1:]]))
    assert times[False] < 4 * times[True], times
