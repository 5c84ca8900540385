"""No garbage collection inside a graph capture: destroying another executor's graphs ends it."""
import contextlib
import gc

import pytest
import torch

from cubic_serve_b200.executor.gpu_executor import capturing


@pytest.mark.parametrize("collects", [True, False])
def test_collection_waits_for_the_capture(monkeypatch, collects):
    monkeypatch.setattr(torch.cuda, "graph", lambda g, stream: contextlib.nullcontext())
    was = gc.isenabled()
    try:
        (gc.enable if collects else gc.disable)()
        with capturing(None, None):
            assert not gc.isenabled()
        assert gc.isenabled() == collects
        with pytest.raises(RuntimeError), capturing(None, None):
            raise RuntimeError
        assert gc.isenabled() == collects
    finally:
        (gc.enable if was else gc.disable)()
