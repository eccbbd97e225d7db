"""Scratch that lives across steps: how it grows, and what is left when it cannot."""
import pytest
import torch

from vlrf_b200.parts.context import Workspace


def test_buffers_that_must_not_double_take_what_is_asked_for():
    ws = Workspace("cpu")
    ws.get("small", 1, 1000, torch.float32)
    ws.get("small", 1, 1500, torch.float32)
    assert ws.bytes() == 4 * 2000
    ws.get("large", 1, 1000, torch.float32, exact=True)
    ws.get("large", 1, 1500, torch.float32, exact=True)
    assert ws.bytes() == 4 * (2000 + 1500)
    generation = ws.generation
    view = ws.get("large", 1, 1200, torch.float32, exact=True)
    assert view.shape == (1, 1200) and ws.bytes() == 4 * 3500 and ws.generation == generation
    ws.frozen = True
    with pytest.raises(RuntimeError):
        ws.get("large", 1, 1600, torch.float32, exact=True)
    assert ws.get("large", 1, 1500, torch.float32).shape == (1, 1500)


def test_a_buffer_that_cannot_grow_is_given_back_first(monkeypatch):
    """The old buffer is not held beside the new one; a failure leaves no view of it, and captured steps see that it went."""
    ws = Workspace("cpu")
    ws.get("large", 1, 1000, torch.float32, exact=True)
    generation, real = ws.generation, torch.empty
    held = []

    def full(*a, **k):
        held.append(ws.bytes())
        raise torch.OutOfMemoryError("no room")
    monkeypatch.setattr(torch, "empty", full)
    with pytest.raises(torch.OutOfMemoryError):
        ws.get("large", 1, 2000, torch.float32, exact=True)
    monkeypatch.setattr(torch, "empty", real)
    assert held == [0] and ws.generation > generation and ws.bytes() == 0
    assert ws.get("large", 1, 1000, torch.float32, exact=True).shape == (1, 1000)
