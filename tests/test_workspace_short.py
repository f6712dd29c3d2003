"""Scratch that cannot be had: the smaller request is taken where the caller names one, and the larger one is
not tried again until the buffers are given back."""
from __future__ import annotations

import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib


@pytest.fixture
def ws(monkeypatch):
    monkeypatch.setattr(_lib, "stream_handle", lambda device: 7)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return _lib._Workspace()


def test_smaller_request(monkeypatch, ws):
    dev, empty, asked = torch.device("cpu", 0), torch.empty, []

    def limited(n, **kw):
        asked.append(n)
        if n > 5000:
            raise torch.OutOfMemoryError("no memory")
        return empty(n, **kw)

    monkeypatch.setattr(torch, "empty", limited)
    with pytest.raises(torch.OutOfMemoryError):
        ws.get(dev, 9000)
    with pytest.raises(torch.OutOfMemoryError):
        ws.get(dev, 9000, 8000)
    small = ws.get(dev, 9000, 1000)
    assert small.numel() == 1000
    n = len(asked)
    assert ws.get(dev, 9000, 900) is small and ws.get(dev, 12000, 1000) is small
    assert len(asked) == n  # the request that failed is not repeated
    assert ws.get(dev, 4000, 1000).numel() == 4000
    ws.clear()
    monkeypatch.setattr(torch, "empty", empty)
    assert ws.get(dev, 9000, 1000).numel() == 9000
