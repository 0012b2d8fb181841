"""Batch.reduce on the host side: which entry point it calls. No GPU: the library is a fake."""
import ctypes
from types import SimpleNamespace

import pytest

from pfc_models_b200 import simulation
from pfc_models_b200.simulation import Batch


class _Plan:
    def __init__(self, handle):
        self.handle = ctypes.c_void_p(handle)

    def reduce(self, out):
        if not self.handle.value:
            raise RuntimeError("null plan")
        out.append(self.handle.value)


def _batch(monkeypatch, handle, plans):
    calls = []
    monkeypatch.setattr(simulation, "_ptr", lambda out: None)
    monkeypatch.setattr(simulation, "_stream_ptr", lambda *a: None)
    b = object.__new__(Batch)
    b.handle, b.plans, b.torch, b.device = ctypes.c_void_p(handle), plans, None, None
    b.lib = SimpleNamespace(pfc_batch_reduce=lambda *a: calls.append(a) or 0, pfc_batch_destroy=lambda h: 0)
    return b, calls


def test_batch_reduce_leaves_closed_plans_and_batches_alone(monkeypatch):
    """Every plan and the batch open: one call. A plan closed: its own refusal, before any launch
    that would read its freed buffers. The batch closed: its plans reduce one by one."""
    b, calls = _batch(monkeypatch, 7, [_Plan(1), _Plan(2)])
    b._reduce_call([])
    assert len(calls) == 1
    b, calls = _batch(monkeypatch, 7, [_Plan(1), _Plan(None)])
    with pytest.raises(RuntimeError, match="null plan"):
        b._reduce_call([[], []])
    assert not calls
    b, calls = _batch(monkeypatch, None, [_Plan(1), _Plan(2)])
    out = [[], []]
    b._reduce_call(out)
    assert out == [[1], [2]] and not calls
