"""Resident engines of many small meshes among a few larger ones: the refit's passes find the
meshes that have work for them, and do not go over the others one by one."""
import numpy as np
import pytest
import torch


def _soup(g, meshes, faces, cuda, spread=0.5, dtype=torch.float64):
    x0 = torch.rand((meshes, faces, 1, 3), generator=g, device=cuda, dtype=dtype) * spread
    x0 = x0 + torch.rand((meshes, faces, 3, 3), generator=g, device=cuda, dtype=dtype) * 0.3
    return x0, x0 + 0.1 * torch.randn((meshes, faces, 3, 3), generator=g, device=cuda, dtype=dtype)


def _engine(soups, **kw):
    from cccollisions_b200.engine import Engine
    sizes = [len(x0) for x0, _ in soups]
    eng = Engine(tri_capacity=sum(sizes), mesh_capacity=len(sizes), **kw)
    sids = [eng.add_mesh(f) for f in sizes]
    for sid, (x0, x1) in zip(sids, soups):
        eng.upload_soup(sid, x0, x1)
    eng.set_active(sids)
    eng.build(sids)
    return eng, sids


def _ordered(rows, times):
    a = np.concatenate([rows.double().cpu().numpy(), times.double().reshape(-1, 1).cpu().numpy()], 1)
    return a[np.lexsort(a.T[::-1])]


@pytest.mark.gpu
@pytest.mark.parametrize("faces,count,larger", [
    (2, 300, {0: 600, 36: 257, 37: 1500, 38: 129, 299: 700}),
    (12, 3000, {5: 300, 1999: 130, 2000: 5000, 2001: 127, 2999: 256}),
    (90, 700, {1: 258, 698: 2000}),
    (2, 45000, {44999: 2000}),                              # beyond a block's look at the next meshes
    (12, 60, {7: 40000, 30: 600, 44: 28000}),               # too large for a team of threads, among many
])
def test_rows_of_each_mesh(cuda, faces, count, larger):
    import cccollisions_b200 as C
    g = torch.Generator(device=cuda).manual_seed(count)
    small = _soup(g, count, faces, cuda)
    soups = [(small[0][i], small[1][i]) for i in range(count)]
    for i, f in larger.items():
        x0, x1 = _soup(g, 1, f, cuda, spread=max(4.0, 0.5 * f ** (1 / 3)))
        soups[i] = (x0[0], x1[0])
    with torch.cuda.device(cuda):
        eng, sids = _engine(soups, max_candidates_per_triangle=32, max_collisions_per_triangle=64)
        eng.ccd()
        st = eng.state(sids)
        assert st["status"] == 0
        total = sum(st["rows"])
        rows = torch.empty((total, 3), dtype=torch.int64, device=cuda)
        times = torch.empty(total, dtype=torch.float64, device=cuda)
        meta = torch.empty(2 * count + 2, dtype=torch.int32, device=cuda)
        eng.pack_rows(rows, times, meta)
        at = meta.tolist()
        mine = {sid: (rows[at[k]:at[k + 1]], times[at[k]:at[k + 1]]) for k, sid in enumerate(at[count + 1:2 * count + 1])}
        eng.close()
    expect = {}
    boxes, tree = C.bvh_motion(*small)
    r, t = C.find_collisions_continuous(boxes, tree, *small, 32, 64)
    r, t = r.cpu(), t.cpu()
    for i, sid in enumerate(sids):
        if i in larger:
            x0, x1 = (x[None] for x in soups[i])
            rr, tt = C.find_collisions_continuous(*C.bvh_motion(x0, x1), x0, x1, 32, 64)
            rr, tt = rr[0].cpu(), tt[0].cpu()
        else:
            rr, tt = r[i], t[i]
        n = int((rr[:, 0] >= 0).sum())
        assert len(mine[sid][0]) == n, i
        if n:
            assert np.array_equal(_ordered(*mine[sid]), _ordered(rr[:n], tt[:n])), i
        expect[sid] = n
    assert sum(expect.values()) == total and total > 0


def _step_times(cuda, meshes=20000, faces=12):
    """Kernel times of a step (20,000 meshes of 12 triangles: none has a node above the refit's
    blocks)."""
    from cccollisions_b200 import _native as N
    g = torch.Generator(device=cuda).manual_seed(1)
    x0, x1 = (x.cpu() for x in _soup(g, meshes, faces, cuda, spread=3.0))
    with torch.cuda.device(cuda):
        eng, _ = _engine(list(zip(x0, x1)), max_candidates_per_triangle=16, max_collisions_per_triangle=8)
        for _ in range(3):
            eng.ccd()
        torch.cuda.synchronize()
        N.timing_begin()
        for _ in range(9):
            eng.ccd()
        torch.cuda.synchronize()
        times = N.timing_end()
        eng.close()
    return {name: ms / count for name, (ms, count) in times.items()}


@pytest.mark.gpu
@pytest.mark.parametrize("meshes,faces", [(20000, 12), (1000, 600)])
def test_small_meshes_cost_the_upper_pass_little(cuda, meshes, faces):
    """Going over them in turn took the upper pass 400 us, far longer than the pass that has all
    the work."""
    times = _step_times(cuda, meshes, faces)
    assert times["k_engine_refit_front"] < times["k_engine_refit"]


@pytest.mark.gpu
def test_small_meshes_share_the_refits_blocks(cuda):
    """With a block each, the refit took 160 us, three times as long as the corner classes' hash
    table, which goes over the same triangles with full blocks; with shared ones about as long."""
    times = _step_times(cuda)
    assert times["k_engine_refit"] < 2 * times["k_weld_insert"]


@pytest.mark.gpu
def test_one_large_mesh_has_the_threads_for_its_climbs(cuda):
    """A mesh with more nodes above the refit's blocks than its upper pass holds is finished by
    climbs, and takes as long in an engine for one mesh as in one for many."""
    from cccollisions_b200 import _native as N
    from cccollisions_b200.engine import Engine
    g = torch.Generator(device=cuda).manual_seed(2)
    x0, x1 = (x[0] for x in _soup(g, 1, 400000, cuda, spread=60.0))
    times = []
    with torch.cuda.device(cuda):
        for capacity in (1, 64):
            eng = Engine(tri_capacity=len(x0), mesh_capacity=capacity, max_candidates_per_triangle=4,
                         max_collisions_per_triangle=4)
            sid = eng.add_mesh(len(x0))
            eng.upload_soup(sid, x0, x1)
            eng.set_active([sid])
            eng.build([sid])
            for _ in range(3):
                eng.ccd()
            torch.cuda.synchronize()
            N.timing_begin()
            for _ in range(9):
                eng.ccd()
            torch.cuda.synchronize()
            times.append(N.timing_end()["k_engine_refit_front"][0])
            eng.close()
    assert times[0] < 1.5 * times[1], times
