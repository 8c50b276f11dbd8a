"""Trees of batches with so many small meshes that several share a block of the build."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("batch,faces", [(2, 2), (149, 128), (300, 65), (1001, 33), (5000, 32), (40000, 2), (40001, 3),
                                         (700, 257), (300, 8193), (149, 16385)])
def test_a_batch_has_the_trees_of_its_meshes(cuda, batch, faces, dtype):
    import cccollisions_b200 as C
    g = torch.Generator(device=cuda).manual_seed(batch + faces)
    x0 = torch.randn((batch, faces, 3, 3), generator=g, device=cuda, dtype=dtype)
    x1 = x0 + 0.1 * torch.randn((batch, faces, 3, 3), generator=g, device=cuda, dtype=dtype)
    boxes, tree = C.bvh_motion(x0, x1)
    # every node's box is the union of its triangles' (min and max are exact), the topology is
    # that of one mesh, which the oracle has tested
    one_boxes, one_tree = C.bvh_motion(x0[:1], x1[:1])
    assert torch.equal(tree, one_tree.expand_as(tree))
    assert torch.equal(boxes[:1], one_boxes)
    both = torch.cat([x0, x1], 2)
    leaves = torch.cat([both.amin(2), both.amax(2)], 2)
    assert torch.equal(boxes[:, faces - 1:], leaves)
    left, right = (boxes[:, one_tree[0, :faces - 1, s]] for s in (1, 2))
    union = torch.cat([torch.minimum(left, right)[..., :3], torch.maximum(left, right)[..., 3:]], 2)
    assert torch.equal(boxes[:, :faces - 1], union)


def _median_ms(fn, turns=9):
    times = []
    for _ in range(turns + 2):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b))
    return float(np.median(times[2:]))


@pytest.mark.gpu
def test_tiny_meshes_cost_about_what_their_triangles_do(cuda):
    """2^20 meshes of two triangles against one mesh of 2^21: a block a mesh takes ten times as
    long, shared blocks about as long; both are large against the launch."""
    import cccollisions_b200 as C
    x = torch.randn((1 << 20, 2, 3, 3), device=cuda)
    one = x.reshape(1, 1 << 21, 3, 3)
    assert _median_ms(lambda: C.bvh(x)) < 5 * _median_ms(lambda: C.bvh(one))
