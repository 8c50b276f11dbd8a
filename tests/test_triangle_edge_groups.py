"""The triangle-edge queries where the kernel's groups of five pairs a warp change behaviour:
no pair that meets, part of a group, whole groups, every lane's pair, and more than one warp."""
from collections import Counter

import numpy as np
import pytest
import torch


def _crossings(n, seed):
    """n pairs of triangles that cross (some sharing one corner), apart from one another."""
    g = np.random.default_rng(seed)
    a = np.array([[0.0, 0, 0], [1, 0, 0], [0, 1, 0]])
    b = np.array([[0.25, 0.25, -1], [0.25, 0.25, 1], [0.25, 2, 0]])
    tri = np.concatenate([np.stack([a, b]) + g.uniform(-0.05, 0.05, (2, 3, 3)) + [5.0 * k, 0, 0] for k in range(n)])
    tri[1::6, 0] = tri[0::6, 2][:len(tri[1::6])]
    return tri


def _soup(f, seed):
    return np.random.default_rng(seed).uniform(0, 1, (f, 3, 3))


MESHES = [("crossings", n) for n in (1, 4, 5, 6, 30, 32, 33, 200)] + [("soup", n) for n in (2, 9, 60)]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind,n", MESHES)
def test_triangle_edge_groups(cuda, oracle, kind, n, dtype):
    import cccollisions_b200 as C
    from cccollisions_b200 import _native as N
    x = (_crossings if kind == "crossings" else _soup)(n, 4).astype(dtype)
    bb, tr = oracle.bvh(x)
    X = torch.from_numpy(x[None]).to(cuda)
    with N.math_library(N.LIB_PORTABLE):
        boxes, tree = C.bvh(X)
        mc = 6 * len(x)
        rows, coefs = C.find_triangle_edge_collisions(boxes, tree, X, 0.0, mc)
        cand = C.find_triangle_edge_candidates(boxes, tree, X, 0.0, mc)
        pairs, masks = C.find_triangle_edge_candidates2(boxes, tree, X, 0.0, mc)
    counted = lambda *cols: Counter(zip(*([tuple(np.ravel(v).tolist()) for v in c] for c in cols)))
    kept = lambda r, *more: [v[0][(r[0, :, 0] >= 0)].cpu().numpy() for v in (r, *more)]
    er, ec = oracle.triangle_edge_collisions(bb, tr, x)
    assert counted(*kept(rows, coefs)) == counted(er, ec)
    cand = cand[0] if isinstance(cand, (list, tuple)) else cand
    assert counted(*kept(cand)) == counted(oracle.triangle_edge_candidates(bb, tr, x))
    assert counted(*kept(pairs, masks)) == counted(*oracle.triangle_edge_candidates2(bb, tr, x))
    if kind == "crossings":
        assert len(oracle.triangle_edge_candidates2(bb, tr, x)[0]) == n
