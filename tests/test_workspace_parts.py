"""Workspace.parts: several buffers in one allocation."""
import torch

from lyapunov_engine_b200.engine.runtime import Workspace


def test_parts_lie_apart_in_one_buffer_and_are_kept():
    ws = Workspace("cpu")
    a, b, c = ws.parts("x", ((3, 5), (7,), (2, 2)), torch.float32)
    assert a.shape == (3, 5) and b.shape == (7,) and c.shape == (2, 2) and len(ws._buffers) == 1
    for i, t in enumerate((a, b, c)):
        assert t.data_ptr() % 16 == a.data_ptr() % 16 and t.is_contiguous()
        t.fill_(i)
    assert [float(t.mean()) for t in (a, b, c)] == [0.0, 1.0, 2.0]
    again = ws.parts("x", ((3, 5), (7,), (2, 2)), torch.float32)
    assert all(t.data_ptr() == s.data_ptr() for t, s in zip((a, b, c), again))
    # a larger set moves the buffer, and what was handed out of the old one is made anew
    ws.parts("x", ((300, 5), (7,)), torch.float32)
    moved = ws.parts("x", ((3, 5), (7,), (2, 2)), torch.float32)
    whole = ws._buffers[("x", torch.float32)]
    assert moved[0].data_ptr() == whole.data_ptr() and moved[2].data_ptr() < whole.data_ptr() + whole.numel() * 4
    assert ws.bytes() == whole.numel() * 4


def test_parts_of_two_byte_types_start_on_16_bytes():
    a, b = Workspace("cpu").parts("x", ((3,), (5,)), torch.bfloat16)
    assert b.data_ptr() - a.data_ptr() == 16
