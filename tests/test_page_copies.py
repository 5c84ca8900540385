"""Page copies of an executor reach the layers that have pages (host side: the launches are recorded, not made)."""
import contextlib
from types import SimpleNamespace

import pytest
import torch

from cubic_serve_b200.executor.gpu_executor import GpuExecutor
from cubic_serve_b200.ops import kernels as K


@pytest.mark.parametrize("pages", [[4, 4], [0, 0, 0, 4, 0, 4], [0]])
def test_layers_without_pages_are_left_out(monkeypatch, pages):
    made = []
    monkeypatch.setattr(K, "copy_pages", lambda cache, src, dst: made.append((cache.shape[0], src.tolist(), dst.tolist())))
    monkeypatch.setattr(torch.cuda, "stream", lambda _: contextlib.nullcontext())
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda *_: None)
    ex = GpuExecutor.__new__(GpuExecutor)
    ex.device, ex.stream = torch.device("cpu"), None
    ex.runner = SimpleNamespace(kv=[torch.zeros(n, 2, 64, dtype=torch.uint8) for n in pages])
    ex.copy_pages([(0, 2), (1, 3)])
    assert made == [(4, [0, 1], [2, 3])] * pages.count(4)
    made.clear()
    ex.copy_pages([])
    assert not made
