"""A caller's tree whose parent column is broken is refused, also when its children are those of
bvh's own trees, for which the rightmost leaves need no climb."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("batch,faces,row", [(1, 2, "leaf")] + [(b, f, row) for b, f in ((2, 3), (2, 40), (1, 1000))
                                                                for row in ("leaf", "internal")])
@pytest.mark.parametrize("parent", [-1, "past the internal nodes"])
def test_broken_parents_are_refused(cuda, batch, faces, row, parent):
    import warnings

    import cccollisions_b200 as C
    g = torch.Generator(device=cuda).manual_seed(faces)
    x0 = torch.rand((batch, faces, 3, 3), generator=g, device=cuda)
    x1 = x0 + 0.01 * torch.rand((batch, faces, 3, 3), generator=g, device=cuda)
    mass = torch.ones((batch, faces, 3), device=cuda)
    check = torch.ones((batch, faces), dtype=torch.bool, device=cuda)
    boxes, tree = C.bvh_motion(x0, x1)
    calls = [
        lambda t: C.find_collisions(boxes, t, x0, 0.0, faces),
        lambda t: C.find_proximity(boxes, t, x0, 0.01, faces),
        lambda t: C.find_collisions_continuous(boxes, t, x0, x1, faces, faces),
        lambda t: C.find_collisions_continuous_partial(boxes, t, x0, x1, check, faces, faces),
        lambda t: C.find_mincol_cand(boxes, t, x0, x1, faces),
        lambda t: C.find_triangle_edge_candidates2(boxes, t, x0, 0.0, faces),
        lambda t: C.compute_impulses(boxes, t, x0, x1, mass, faces, faces),
    ]
    at = faces - 1 + faces // 2 if row == "leaf" else (faces - 1) // 2 or 1
    broken = tree.clone()
    broken[batch - 1, at, 0] = parent if parent == -1 else faces - 1
    for call in calls:
        with warnings.catch_warnings():
            warnings.simplefilter("ignore")          # (rows past the capacity)
            call(tree)
            with pytest.raises(RuntimeError, match="malformed tree"):
                call(broken)
