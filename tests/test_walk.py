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


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [
    [(129, 2), (130, 2), (17, 17), (257, 2), (33, 17)],      # 256 to 1,024 triangles: no or few nodes above a block
    [(60, 50), (3, 2), (331, 341), (20, 15)],                # 224,400: more of them than one block of threads holds
])
def test_refit_above_the_blocks(cuda, sizes):
    """Rows of the resident meshes against the per-call path, as built and after the positions
    changed (a refit only)."""
    import cccollisions_b200 as C
    from cccollisions_b200 import workloads as W
    from cccollisions_b200.engine import Engine

    def ordered(rows, times):
        a = np.concatenate([rows.double().cpu().numpy(), times.double().reshape(-1, 1).cpu().numpy()], 1)
        return a[np.lexsort(a.T[::-1])]

    with torch.cuda.device(cuda):
        meshes = [W.jittered_fold(i, nx, ny, noise=0.5 / nx, drop=0.5 / nx)[:2] for i, (nx, ny) in enumerate(sizes)]
        total = sum(len(x0) for x0, _ in meshes)
        eng = Engine(tri_capacity=total, mesh_capacity=len(meshes), max_candidates_per_triangle=64,
                     max_collisions_per_triangle=32)
        sids = [eng.add_mesh(len(x0)) for x0, _ in meshes]
        for turn in range(2):
            if turn:
                meshes = [(x0[:, :, [1, 0, 2]] * 1.5, x1[:, :, [1, 0, 2]] * 1.5) for x0, x1 in meshes]
            for sid, (x0, x1) in zip(sids, meshes):
                eng.upload_soup(sid, x0, x1)
            if turn == 0:
                eng.set_active(sids)
                eng.build(sids)
            eng.ccd()
            st = eng.state(sids)
            assert st["status"] == 0
            for sid, (x0, x1), n in zip(sids, meshes, st["rows"]):
                X0, X1 = (torch.from_numpy(np.ascontiguousarray(x)[None]).to(cuda) for x in (x0, x1))
                rows, times = C.find_collisions_continuous(*C.bvh_motion(X0, X1), X0, X1, 64, 32)
                there = rows[0, :, 0] >= 0
                assert n == int(there.sum())
                assert np.array_equal(ordered(*eng.collisions(sid, int(n))), ordered(rows[0][there], times[0][there]))
        eng.close()
