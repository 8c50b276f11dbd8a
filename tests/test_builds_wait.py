"""bvh and bvh_motion return when their tensors are complete, like the queries, so that a caller
may build on one stream and query on another."""
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("motion", [False, True])
def test_a_build_is_complete_when_the_call_returns(cuda, motion):
    import cccollisions_b200 as C
    from cccollisions_b200 import api
    x0 = torch.rand((1, 1000, 3, 3), device=cuda)
    x1 = x0 + 0.01
    build = (lambda: C.bvh_motion(x0, x1)) if motion else (lambda: C.bvh(x0))
    build()                                          # (the library and the allocator are warm)
    side = torch.cuda.Stream(cuda)
    torch.cuda.synchronize(cuda)
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)                # some 10 ms ahead of the build
        build()
        assert side.query()
    assert api.CHECK_STATUS
    api.CHECK_STATUS = False
    try:
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)
            build()
            assert not side.query()                  # left to the caller's stream
    finally:
        api.CHECK_STATUS = True
        torch.cuda.synchronize(cuda)
