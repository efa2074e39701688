"""Host-side parts of the functional front end that need no device."""
import torch

from multitokenatention_triton_b200 import ops


def test_copies_of_unaligned_planes_are_left_out_when_there_is_no_room(monkeypatch):
    x = torch.zeros(1, 4, 1025, 1025, dtype=torch.bfloat16)
    assert ops._row_copies(x).numel() >= 2 * 4 * 1025 * 1040 * 2

    def empty(*a, **k):
        raise torch.cuda.OutOfMemoryError("no room")

    monkeypatch.setattr(torch, "empty", empty)
    assert ops._row_copies(x) is None
