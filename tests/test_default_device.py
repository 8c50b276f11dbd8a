"""Calls do not depend on torch's default device, in any thread."""
import threading

import pytest
import torch


def _first_call(device, x0, x1, out):
    import cccollisions_b200 as C
    try:
        torch.set_default_device(device)             # (of this thread)
        boxes, tree = C.bvh_motion(x0, x1)
        out.append(C.find_collisions(boxes, tree, x0, 0.0, 100))
    except Exception as exc:                         # noqa: BLE001 - handed to the test's thread
        out.append(exc)
    finally:
        torch.set_default_device(None)


@pytest.mark.gpu
@pytest.mark.parametrize("device", ["cuda", "meta", "cpu"])
def test_a_threads_first_call_under_a_default_device(cuda, device):
    x0 = torch.rand((1, 100, 3, 3), device=cuda)
    x1 = x0 + 0.01
    out = []
    for default in (None, device):
        # a new thread: whatever a call keeps for its thread is made in it
        t = threading.Thread(target=_first_call, args=(default, x0, x1, out))
        t.start()
        t.join()
    assert all(isinstance(o, torch.Tensor) for o in out), out
    there = [torch.unique(o[0][o[0, :, 0] >= 0], dim=0) for o in out]
    assert torch.equal(*there)
