"""bvh / bvh_motion against the oracle at the sizes where the build's levels and launches end."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("batch,faces", [(3, 2), (2, 3), (1, 33), (2, 255), (1, 256), (2, 257), (1, 2049), (1, 65537),
                                         (1, 262145)])
def test_build_at_the_edges_of_its_blocks(cuda, oracle, batch, faces, dtype):
    import cccollisions_b200 as C
    rng = np.random.default_rng(faces)
    x0 = rng.normal(0, 1, (batch, faces, 3, 3)).astype(dtype)
    x1 = (x0 + rng.normal(0, 0.1, x0.shape)).astype(dtype)
    X0, X1 = torch.from_numpy(x0).to(cuda), torch.from_numpy(x1).to(cuda)
    for got, motion in ((C.bvh(X0), False), (C.bvh_motion(X0, X1), True)):
        for b in range(batch):
            boxes, tree = oracle.bvh(x0[b], x1[b] if motion else None)
            assert np.array_equal(got[0][b].cpu().numpy(), boxes)
            assert np.array_equal(got[1][b].cpu().numpy(), tree)


def _query(lib, boxes, tree, x0, x1, mask, narrow_nodes):
    """(status, candidates, sorted rows with times) of one continuous query with all of its
    scratch or with just enough for the binary nodes."""
    import ctypes

    from cccollisions_b200 import _native as N
    B, F = x0.shape[:2]
    p = lambda t: None if t is None else ctypes.c_void_p(t.data_ptr())
    size = lib.ccc_workspace_size(N.OP_CONTINUOUS, B, F, F)
    if narrow_nodes:
        size -= max(0, (64 * B * F // 256 - 1) * 256)
    ws = torch.full((size,), 0xAB, dtype=torch.uint8, device=x0.device)
    rows = torch.full((B, F * F, 3), -1, dtype=torch.int64, device=x0.device)
    times = torch.full((B, F * F, 1), -1, dtype=x0.dtype, device=x0.device)
    assert lib.ccc_find_collisions_continuous(int(x0.dtype == torch.float64), p(boxes), p(tree), p(x0), p(x1), p(mask),
                                              B, F, F, F, p(rows), p(times), p(ws), size, None) == 0
    out = (ctypes.c_int32 * 4)()
    assert lib.ccc_read_counters(p(ws), out, None) == 0
    got = torch.cat([rows.double(), times.double()], 2).cpu().numpy()
    return out[0], out[1], [sorted(map(tuple, b[b[:, 0] >= 0])) for b in got]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("batch,nx,ny", [(1, 2, 2), (3, 9, 7), (2, 17, 12)])
def test_wide_nodes_give_the_binary_nodes_pairs(cuda, native_lib, oracle, batch, nx, ny, dtype):
    """The four-wide import and walk against the binary ones: trees of bvh_motion and of a
    spatial sort, boxes that do not contain their children's, NaN and infinite boxes, masks."""
    import cccollisions_b200 as C
    from cccollisions_b200 import workloads as W
    parts = [W.jittered_fold(seed, nx, ny, dtype=dtype) for seed in range(batch)]
    x0, x1 = (torch.from_numpy(np.stack([p[k] for p in parts])).to(cuda) for k in (0, 1))
    F = x0.shape[1]
    rng = np.random.default_rng(F)
    boxes, tree = C.bvh_motion(x0, x1)
    spatial = [oracle.bvh(p[0], p[1], spatial=True) for p in parts]
    shrunk, odd = boxes.clone(), boxes.clone()
    some = torch.from_numpy(rng.random((batch, F - 1)) < 0.2).to(cuda)
    shrunk[:, :F - 1][some] *= 0.5
    odd[:, F - 1 + F // 2] = float("nan")
    odd[:, F // 3] = float("inf")
    masks = [None] + [torch.from_numpy((rng.random((batch, F)) < share).astype(np.uint8)).to(cuda)
                      for share in (0.0, 0.3, 1.0)]
    for bb, tr in ((boxes, tree), tuple(torch.from_numpy(np.stack(t)).to(cuda) for t in zip(*spatial)),
                   (shrunk, tree), (odd, tree)):
        for mask in masks:
            wide = _query(native_lib, bb, tr, x0, x1, mask, False)
            assert wide == _query(native_lib, bb, tr, x0, x1, mask, True)
            assert wide[0] == 0
