"""The tree walk emits every pair of overlapping boxes once, at the sizes where its warps'
shared stack, leaf queue and output buffer change behaviour."""
import numpy as np
import pytest
import torch


def _overlapping_pairs(x):
    lo, hi = x.min(1), x.max(1)
    hit = np.ones((len(x), len(x)), bool)
    for c in range(3):
        hit &= (lo[:, None, c] <= hi[None, :, c]) & (hi[:, None, c] >= lo[None, :, c])
    return int(np.triu(hit, 1).sum())


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,spread", [
    ((2,), 0.0), ((2, 3, 2), 0.0),             # the smallest trees
    ((31, 33, 64, 5), 0.1),                    # groups that span meshes
    ((1500,), 0.0),                            # every box meets every other: the stack fills up
    ((700, 3, 900), 0.02),
    ((6000, 2, 4097), 5.0),                    # sparse: most visits end high in the tree
])
def test_walk_finds_every_overlapping_pair(cuda, sizes, spread):
    from cccollisions_b200.engine import Engine
    rng = np.random.default_rng(len(sizes) + sum(sizes))
    meshes = [(rng.uniform(0, 1, (f, 3, 3)) + spread * rng.uniform(0, 10, (f, 1, 3))).astype(np.float32)
              for f in sizes]
    expect = sum(_overlapping_pairs(x) for x in meshes)
    maxc = max(sizes)
    with torch.cuda.device(cuda):
        eng = Engine(tri_capacity=sum(sizes), mesh_capacity=len(sizes), max_candidates_per_triangle=maxc,
                     max_collisions_per_triangle=1, dtype=torch.float32)
        sids = [eng.add_mesh(f) for f in sizes]
        for sid, x in zip(sids, meshes):
            eng.upload_soup(sid, x, x)         # nothing moves: no sub-test has a root
        eng.set_active(sids)
        eng.build(sids)
        # the triangles share no vertex, so no pair is dropped, and fp32 boxes are exact
        for choice, s in enumerate(Engine.schedules()):
            if s["warp_traversal"] == 0 and s["staged_levels"] == 0 and s["narrow_batch"] == 1:
                eng.set_schedule(choice)
                eng.ccd()
                got = eng.counters()
                assert got["status"] == 0
                assert got["candidates"] == expect
        eng.close()
