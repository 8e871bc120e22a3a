"""A grid that is not on a GPU has no stream to run on: asking for one raises
before any pointer reaches the engine (as torch's own query does)."""
import pytest
import torch

from gbstencil import grid


def test_no_stream_for_a_host_grid(monkeypatch):
    monkeypatch.setattr(grid, "_raw_stream", lambda index: 0)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)
    with pytest.raises((ValueError, RuntimeError)):
        grid.current_stream(torch.device("cpu"))
