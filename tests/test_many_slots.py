"""Continuous queries on batches around 2^24 triangles: up to there a pair's sub-test mask is kept
in the pair's own words, beyond it in an array of its own."""
import ctypes

import numpy as np
import pytest
import torch

PER_TRIANGLE = 4                 # rows; a mesh is two triangles


def _pairs(g, count, dtype, cuda):
    """Meshes of two triangles that cross or pass each other."""
    x0 = torch.rand((count, 2, 3, 3), generator=g, device=cuda, dtype=torch.float64)
    x1 = x0 + 0.8 * torch.randn((count, 2, 1, 3), generator=g, device=cuda, dtype=torch.float64)
    x1 = x1 + 0.1 * torch.randn((count, 2, 3, 3), generator=g, device=cuda, dtype=torch.float64)
    return x0.to(dtype), x1.to(dtype)


def _scratch(lib, op, B, device):
    return torch.full((lib.ccc_workspace_size(op, B, 2, 1),), 0xAB, dtype=torch.uint8, device=device)


def _ok(lib, ws):
    out = (ctypes.c_int32 * 4)()
    assert lib.ccc_read_counters(ws.data_ptr(), out, torch.cuda.current_stream().cuda_stream) == 0
    return list(out)


def _rows(lib, x0, x1, per):
    """Each mesh's sub-tests and times, sorted, as 16 k + time (-1: no row); the status and counters."""
    import cccollisions_b200 as C
    from cccollisions_b200 import _native as N
    B = x0.shape[0]
    boxes, tree = C.bvh_motion(x0, x1)
    ws = _scratch(lib, N.OP_CONTINUOUS, B, x0.device)
    rows = torch.full((B, 2 * per, 3), -1, dtype=torch.int64, device=x0.device)
    times = torch.full((B, 2 * per), -1.0, dtype=x0.dtype, device=x0.device)
    assert lib.ccc_find_collisions_continuous(int(x0.dtype == torch.float64), boxes.data_ptr(), tree.data_ptr(),
                                              x0.data_ptr(), x1.data_ptr(), None, B, 2, 1, per, rows.data_ptr(),
                                              times.data_ptr(), ws.data_ptr(), ws.numel(),
                                              torch.cuda.current_stream().cuda_stream) == 0
    status = _ok(lib, ws)
    there = rows[:, :, 0] >= 0
    assert bool((there == ((rows[:, :, 0] == 0) & (rows[:, :, 1] == 1))).all())
    key = torch.where(there, 16.0 * rows[:, :, 2] + times.double(), -1.0)
    return torch.sort(key, 1)[0], there.sum(1), status


def _impulses(lib, x0, x1, mass):
    import cccollisions_b200 as C
    from cccollisions_b200 import _native as N
    B = x0.shape[0]
    boxes, tree = C.bvh_motion(x0, x1)
    ws = _scratch(lib, N.OP_IMPULSES, B, x0.device)
    dv, dx = (torch.zeros((B, 2, 3, 3), dtype=x0.dtype, device=x0.device) for _ in range(2))
    count = torch.zeros((B, 2, 3), dtype=torch.int32, device=x0.device)
    assert lib.ccc_compute_impulses(int(x0.dtype == torch.float64), boxes.data_ptr(), tree.data_ptr(), x0.data_ptr(),
                                    x1.data_ptr(), mass.data_ptr(), None, B, 2, 1, PER_TRIANGLE, dv.data_ptr(), dx.data_ptr(),
                                    count.data_ptr(), ws.data_ptr(), ws.numel(),
                                    torch.cuda.current_stream().cuda_stream) == 0
    return dv, dx, count, _ok(lib, ws)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("meshes", [1 << 23, (1 << 23) + 1])
def test_every_mesh_has_its_rows_and_impulses(cuda, native_lib, meshes, dtype):
    g = torch.Generator(device=cuda).manual_seed(1)
    with torch.cuda.device(cuda):
        x0, x1 = _pairs(g, 5000, dtype, cuda)
        keys, n, status = _rows(native_lib, x0, x1, 16)
        assert status[0] == 0
        fit = n <= 2 * PER_TRIANGLE
        x0, x1, keys, n = x0[fit].contiguous(), x1[fit].contiguous(), keys[fit][:, -2 * PER_TRIANGLE:], n[fit]
        assert int((n == 0).sum()) > 300 and int((n == 1).sum()) > 100 and int((n > 1).sum()) > 100
        mass = torch.rand((len(x0), 2, 3), generator=g, device=cuda, dtype=torch.float64).to(dtype) + 0.5
        few = _impulses(native_lib, x0, x1, mass)
        assert few[3][0] == 0

        # the same meshes over and over, in any order
        which = torch.randint(0, len(x0), (meshes,), generator=g, device=cuda)
        which[-1] = int(torch.nonzero(n > 1)[0])
        X0, X1 = x0[which], x1[which]
        got, count, status = _rows(native_lib, X0, X1, PER_TRIANGLE)
        assert status[0] == 0
        assert torch.equal(count, n[which])
        assert torch.equal(got, keys[which])
        del got, count

        dv, dx, count, status = _impulses(native_lib, X0, X1, mass[which])
        assert status[0] == 0
        assert torch.equal(count, few[2][which])
        # (a corner with several contacts takes them in any order)
        alone = (few[2][which].amax((1, 2)) <= 1)
        assert int(alone.sum()) > meshes // 4
        assert torch.equal(dv[alone], few[0][which][alone]) and torch.equal(dx[alone], few[1][which][alone])
