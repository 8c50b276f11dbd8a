"""ccc_fill writes its arrays, all of them and nothing beside them, at any 4-byte alignment."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("start", [0, 1, 2, 3])
@pytest.mark.parametrize("words", [0, 1, 3, 4, 5, 1023, 700_001])
def test_fill(cuda, native_lib, start, words):
    patterns = (-1, 0, 0x1122334455667788)
    room = torch.full((3, words + 16), 77, dtype=torch.int32, device=cuda)
    args = []
    for row, pattern in zip(room, patterns):
        part = row[4 + start:4 + start + words]
        args += [part.data_ptr() if words else None, 4 * words, pattern]
    assert native_lib.ccc_fill(*args, torch.cuda.current_stream(cuda).cuda_stream) == 0
    got = room.cpu().numpy()
    for row, pattern in zip(got, patterns):
        halves = np.array([pattern & 0xffffffff, (pattern >> 32) & 0xffffffff], dtype=np.uint32).view(np.int32)
        assert np.array_equal(row[4 + start:4 + start + words], np.resize(halves, words))
        assert (row[:4 + start] == 77).all() and (row[4 + start + words:] == 77).all()


def test_fill_refuses_what_it_cannot_write(native_lib):
    assert native_lib.ccc_fill(None, 8, 0, None, 0, 0, None, 0, 0, None) == 1      # no array
    assert native_lib.ccc_fill(8, 6, 0, None, 0, 0, None, 0, 0, None) == 1         # not whole words
    assert native_lib.ccc_fill(10, 8, 0, None, 0, 0, None, 0, 0, None) == 1        # misaligned
    assert native_lib.ccc_fill(None, -4, 0, None, 0, 0, None, 0, 0, None) == 1
    assert native_lib.ccc_fill(None, 0, 0, None, 0, 0, None, 0, 0, None) == 0
