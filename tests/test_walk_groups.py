"""The tree walk finds every pair of overlapping boxes on both sides of the sizes at which its
warps' groups of queries change: one group a warp, large groups and small ones at the end, and
more than the stack's 32 queries a warp."""
import numpy as np
import pytest
import torch

WARPS = 148 * 8 * 4         # of the engine's default schedule and of the tensor walk


def _overlapping_pairs(x):
    lo, hi = x.amin(1), x.amax(1)
    count = 0
    for at in range(0, len(x), 4096):
        a, b = lo[at:at + 4096, None], hi[at:at + 4096, None]
        count += int(((a <= hi[None]) & (b >= lo[None])).all(-1).sum())
    return (count - len(x)) // 2


@pytest.mark.gpu
@pytest.mark.parametrize("count", [WARPS * 12 - 1, WARPS * 12, WARPS * 12 + 1, WARPS * 16, WARPS * 32 + 5])
def test_every_pair_of_a_soup(cuda, count):
    from cccollisions_b200.engine import Engine
    g = np.random.default_rng(count)
    # more crowded towards one corner
    x = (g.uniform(0, 1, (count, 3, 3)) * 0.02 + g.uniform(0, 1, (count, 1, 3)) ** 1.5).astype(np.float32)
    pairs = _overlapping_pairs(torch.from_numpy(x).to(cuda))
    assert pairs > count // 8
    with torch.cuda.device(cuda):
        eng = Engine(tri_capacity=count, mesh_capacity=1, max_candidates_per_triangle=pairs // count + 2,
                     max_collisions_per_triangle=1, dtype=torch.float32)
        sid = eng.add_mesh(count)
        eng.upload_soup(sid, x, x)
        eng.set_active([sid])
        eng.build([sid])
        eng.ccd()
        got = eng.counters()
        assert got["status"] == 0 and got["candidates"] == pairs
        eng.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(169, 170), (178, 168), (300, 260)])
def test_rows_of_a_call_are_the_engines(cuda, nx, ny):
    """The tensor walk on 56,784, 59,118 and 154,882 triangles against the engine's walk with one
    query a thread."""
    import cccollisions_b200 as C
    from cccollisions_b200 import workloads as W
    from cccollisions_b200.engine import Engine
    x0, x1 = W.jittered_fold(1, nx, ny, noise=0.3 / nx, drop=0.5 / nx)[:2]
    X0, X1 = (torch.from_numpy(x[None]).to(cuda) for x in (x0, x1))
    rows, times = C.find_collisions_continuous(*C.bvh_motion(X0, X1), X0, X1, 48, 32)
    got = torch.cat([rows[0].double(), times[0]], 1)[rows[0, :, 0] >= 0].cpu().numpy()
    with torch.cuda.device(cuda):
        eng = Engine(tri_capacity=len(x0), mesh_capacity=1, max_candidates_per_triangle=48,
                     max_collisions_per_triangle=32)
        sid = eng.add_mesh(len(x0))
        eng.upload_soup(sid, x0, x1)
        eng.set_active([sid])
        eng.build([sid])
        eng.set_schedule(next(i for i, s in enumerate(Engine.schedules()) if s["staged_levels"] == 1))
        eng.ccd()
        st = eng.state([sid])
        assert st["status"] == 0
        r, t = eng.collisions(sid, int(st["rows"][0]))
        want = np.concatenate([r.double().cpu().numpy(), t.double().reshape(-1, 1).cpu().numpy()], 1)
        eng.close()
    order = lambda a: a[np.lexsort(a.T[::-1])]
    assert len(want) > 1000 and np.array_equal(order(got), order(want))
