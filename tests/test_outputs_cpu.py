"""The output tensors of the calculators, without a GPU: what happens around
the allocation that the engine asks for in the middle of a build."""

import ctypes

import pytest
import torch

from vesin_b200 import _outputs


class _Stream:
    def __init__(self, handle, events):
        self.cuda_stream = handle
        self._events = events

    def synchronize(self):
        self._events.append("wait")


@pytest.mark.parametrize("handle, waits", [(0, []), (7, ["wait"])])
def test_engine_waits_for_memory_it_was_handed(handle, waits, monkeypatch):
    """On a stream other than the default one the engine is not ordered behind
    the allocation: the callback waits for the stream after it."""
    events = []
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device: _Stream(handle, events))
    outputs = _outputs.OutputTensors("ijSdD", torch.device("cpu"), torch.int64, torch.float64)
    allocate = outputs.allocate
    monkeypatch.setattr(outputs, "allocate", lambda n: (allocate(n), events.append("allocate")))
    with outputs:
        assert _outputs.allocate_callback(None, 5, ctypes.byref(outputs.arrays)) == 0
    assert events == ["allocate"] + waits
    assert outputs.arrays.capacity == 5 and [len(t) for t in outputs.take(5)] == [5] * 5
