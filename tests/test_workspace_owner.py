"""Scratch handed out for an owner lives and dies with that owner, apart from the streams' buffers."""
from __future__ import annotations

import gc
import threading
import weakref

import pytest
import torch

from jscc_recon_spect_cylinder_gb300 import _lib


@pytest.fixture
def ws(monkeypatch):
    monkeypatch.setattr(_lib, "stream_handle", lambda device: 7)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return _lib._Workspace()


def test_owner(ws):
    class Holder(list):
        pass

    dev, mine, other = torch.device("cpu", 0), Holder(), Holder()
    shared = ws.get(dev, 2000)
    with ws.owned_by(mine):
        a = ws.get(dev, 1000)
        assert a is not shared and ws.get(dev, 500) is a
        big = ws.get(dev, 3000)
        seen = []
        t = threading.Thread(target=lambda: seen.append(ws.get(dev, 1500)))  # another thread is not affected
        t.start()
        t.join()
        assert seen[0] is shared
        with ws.owned_by(other):
            assert ws.get(dev, 1000) is not big
        assert ws.get(dev, 3000) is big
    assert ws.get(dev, 2000) is shared
    first = weakref.ref(a)
    del a
    assert first() is not None  # kernels captured before the growth still use it
    del big, mine
    gc.collect()
    assert first() is None
