"""Scratch memory by tag: views are made once, follow a buffer that grows, and do not pile up. No GPU."""
import pytest
import torch

from llmengine.engine.context import Workspace


def test_views_are_kept_and_follow_the_buffer():
    ws = Workspace(torch.device("cpu"))
    a = ws.get("t", (4, 8), torch.float32)
    assert ws.get("t", (4, 8), torch.float32) is a and ws.get("t", [4, 8], torch.float32) is a
    half = ws.get("t", (4, 8), torch.bfloat16)
    assert half.dtype == torch.bfloat16 and half.data_ptr() == a.data_ptr()
    small = ws.get("t", (2, 8), torch.float32)
    assert small.data_ptr() == a.data_ptr() and ws.bytes() == 256
    big = ws.get("t", (400, 8), torch.float32)
    again = ws.get("t", (4, 8), torch.float32)
    assert again.data_ptr() == big.data_ptr() and again is not a  # nobody is handed the buffer that was given up
    ws.frozen = True
    assert ws.get("t", (400, 8), torch.float32) is big
    with pytest.raises(RuntimeError, match="would have to grow"):
        ws.get("t", (401, 8), torch.float32)


def test_cleared_when_made_or_grown():
    ws = Workspace(torch.device("cpu"))
    z = ws.get_zeroed("z", (8,), torch.int32)
    z.fill_(3)
    assert int(ws.get_zeroed("z", (8,), torch.int32).sum()) == 24
    assert int(ws.get_zeroed("z", (800,), torch.int32).sum()) == 0


def test_views_of_ever_new_sizes_are_bounded():
    ws = Workspace(torch.device("cpu"))
    ws.get("t", (Workspace.MAX_VIEWS + 10,), torch.int32)
    for n in range(1, Workspace.MAX_VIEWS + 10):
        assert ws.get("t", (n,), torch.int32).shape == (n,)
    assert len(ws._views) <= Workspace.MAX_VIEWS and len(ws._buffers) == 1
