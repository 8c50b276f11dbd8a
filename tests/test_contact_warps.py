"""Impulses of listed contacts, which a warp's lanes add together: fewer contacts than a warp,
whole warps, rests, and rows in between that name no triangle or no type."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("count", [1, 31, 32, 33, 127, 700])
@pytest.mark.parametrize("triangles", [2, 40])
def test_impulses_of_listed_rows(cuda, oracle, count, triangles, dtype):
    import cccollisions_b200 as C
    from cccollisions_b200 import _native as N
    g = np.random.default_rng(count + triangles)
    x0 = g.uniform(0, 1, (triangles, 3, 3)).astype(dtype)
    x1 = (x0 + g.normal(0, 0.2, x0.shape)).astype(dtype)
    m = g.uniform(0.5, 2.0, (triangles, 3)).astype(dtype)
    rows = np.stack([g.integers(0, triangles, count), g.integers(0, triangles, count), g.integers(0, 15, count)], 1)
    times = g.uniform(0, 1, count).astype(dtype)
    skipped = g.random(count) < 0.2
    rows[skipped, g.integers(0, 3, int(skipped.sum()))] = -1
    with N.math_library(N.LIB_PORTABLE):
        dv, dx, n = C.compute_impulses_from_collisions(
            *(torch.from_numpy(np.ascontiguousarray(a[None])).to(cuda) for a in (rows, times[:, None], x0, x1, m)))
    edv, edx, en = oracle.impulses_from_rows(x0, x1, m, rows[~skipped], times[~skipped].astype(np.float64))
    assert np.array_equal(n[0].cpu().numpy(), en)
    # sums of up to `count` terms in any order
    tol = count * np.finfo(dtype).eps
    for a, b in ((dv, edv), (dx, edx)):
        a, b = a[0].double().cpu().numpy(), b.astype(np.float64)
        fine = np.isfinite(b)           # (a pair of one triangle with itself gives NaN)
        assert np.array_equal(np.isfinite(a), fine)
        assert np.abs(a - b)[fine].max(initial=0) <= tol * max(np.abs(b)[fine].max(initial=0), 1.0) * 4
