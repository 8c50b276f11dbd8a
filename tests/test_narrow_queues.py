"""The continuous narrow phase against the oracle where its queues, batches and record lists
change behaviour: fewer sub-tests than a batch, a few more, many per pair, and more passing
roots than the list of records holds."""
from collections import Counter

import numpy as np
import pytest
import torch


def _soup(f, seed):
    """f triangles in one unit box, every pair a candidate, moving through one another."""
    g = np.random.default_rng(seed)
    x0 = g.uniform(0, 1, (f, 3, 3))
    return x0, x0 + g.normal(0, 0.5, x0.shape), g.uniform(0.5, 2.0, (f, 3))


def _mesh(name):
    from cccollisions_b200 import workloads as W
    kind, *size = name.split("-")
    return _soup(int(size[0]), 3) if kind == "soup" else W.jittered_fold(5, int(size[0]), int(size[1]))


MESHES = ["soup-2", "soup-7", "soup-40", "soup-90", "fold-3-3", "fold-9-8", "fold-33-31"]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("name", MESHES)
def test_rows_and_impulses(cuda, oracle, name, dtype):
    import cccollisions_b200 as C
    from cccollisions_b200 import _native as N
    x0, x1, m = (a.astype(dtype) for a in _mesh(name))
    F = len(x0)
    X0, X1, M = (torch.from_numpy(a[None]).to(cuda) for a in (x0, x1, m))
    with N.math_library(N.LIB_PORTABLE):
        boxes, tree = C.bvh_motion(X0, X1)
        rows, times = C.find_collisions_continuous(boxes, tree, X0, X1, min(F, 64), 15 * min(F, 64))
        dv, dx, count = C.compute_impulses(boxes, tree, X0, X1, M, min(F, 64))
    bb, tr = oracle.bvh(x0, x1)
    er, et = oracle.ccd(bb, tr, x0, x1)
    n = int((rows[0, :, 0] >= 0).sum())
    got = Counter(zip(map(tuple, rows[0, :n].tolist()), times[0, :n, 0].double().tolist()))
    assert got == Counter(zip(map(tuple, er.tolist()), map(float, et.tolist())))
    edv, edx, ecount, contacts = oracle.impulses(bb, tr, x0, x1, m)
    assert contacts == len(er)
    assert np.array_equal(count[0].cpu().numpy(), ecount)
    tol = 1e-9 if dtype == np.float64 else 2e-3          # sums of up to thousands of terms, in any order
    for a, b in ((dv, edv), (dx, edx)):
        a, b = a[0].double().cpu().numpy(), b.astype(np.float64)
        fine = np.isfinite(b)
        assert np.array_equal(np.isfinite(a), fine)
        assert np.abs(a - b)[fine].sum() <= tol * np.abs(b)[fine].sum() + 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("name", MESHES)
def test_engine_rows_and_loop(cuda, oracle, name):
    """The resident engine with room for no more candidates than there are, so that the roots
    that pass outnumber the record list on the soups."""
    from cccollisions_b200 import _native as N
    from cccollisions_b200.engine import Engine
    x0, x1, m = _mesh(name)
    F = len(x0)
    verts0, faces = np.unique(x0.reshape(-1, 3), axis=0, return_inverse=True)
    faces = faces.reshape(-1, 3).astype(np.int32)
    verts1 = np.empty_like(verts0)
    verts1[faces.ravel()] = x1.reshape(-1, 3)
    bb, tr = oracle.bvh(x0, x1)
    er, et = oracle.ccd(bb, tr, x0, x1)
    maxc = -(-len(oracle.candidates(bb, tr)) // F) + 2
    with torch.cuda.device(cuda), N.math_library(N.LIB_PORTABLE):
        eng = Engine(tri_capacity=F, vert_capacity=len(verts0), mesh_capacity=1, max_candidates_per_triangle=maxc,
                     max_collisions_per_triangle=15 * maxc)
        sid = eng.add_mesh(F, len(verts0))
        eng.upload_mesh(sid, verts0, verts1, verts1 - verts0, faces, m)
        eng.set_active([sid])
        eng.loop_prepare([sid])
        eng.ccd()
        st = eng.state([sid])
        assert st["status"] == 0
        r, t = eng.collisions(sid, int(st["rows"][0]))
        got = Counter(zip(map(tuple, r.tolist()), t.tolist()))
        assert got == Counter(zip(map(tuple, er.tolist()), map(float, et.tolist())))
        eng.loop_step(1)
        assert int(eng.state([sid])["contacts"][0]) == len(er)
        eng.close()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("name,threshold", [(n, t) for n in MESHES for t in (0.0, 0.02, 0.3)])
def test_proximity(cuda, oracle, name, threshold, dtype):
    import cccollisions_b200 as C
    x0 = _mesh(name)[0].astype(dtype)
    F = len(x0)
    X = torch.from_numpy(x0[None]).to(cuda)
    boxes, tree = C.bvh(X)
    (rows,) = C.find_proximity(boxes, tree, X, threshold, 15 * min(F, 400))
    n = int((rows[0, :, 0] >= 0).sum())
    bb, tr = oracle.bvh(x0)
    assert Counter(map(tuple, rows[0, :n].tolist())) == Counter(map(tuple, oracle.proximity(bb, tr, x0, threshold)[0].tolist()))
