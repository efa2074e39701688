"""Host-side parts of the functional front end that need no device."""
import importlib.util
import types

import torch

from multitokenatention_triton_b200 import _lib, ops


def test_copies_of_unaligned_planes_are_left_out_when_there_is_no_room(monkeypatch):
    x = torch.zeros(1, 4, 1025, 1025, dtype=torch.bfloat16)
    assert ops._row_copies(x).numel() >= 2 * 4 * 1025 * 1040 * 2

    def empty(*a, **k):
        raise torch.cuda.OutOfMemoryError("no room")

    monkeypatch.setattr(torch, "empty", empty)
    assert ops._row_copies(x) is None


def test_stream_of_a_torch_without_the_raw_getter(monkeypatch):
    monkeypatch.delattr(torch._C, "_cuda_getCurrentRawStream", raising=False)
    spec = importlib.util.spec_from_file_location("lib_of_another_torch", _lib.__file__)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device: types.SimpleNamespace(cuda_stream=1000 + device.index))
    assert m.stream_ptr(torch.device("cuda", 3)) == 1003
