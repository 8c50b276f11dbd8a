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
