"""The output tensors of the calculators, without a GPU: what happens around
the allocation that the engine asks for in the middle of a build, and the room
that is guessed before it."""

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


def _outputs_of(quantities="ijSdD"):
    return _outputs.OutputTensors(quantities, torch.device("cpu"), torch.int64, torch.float64)


def test_room_follows_the_number_of_points():
    outputs = _outputs_of()
    outputs.allocate_guess((0, 0), 1000)
    assert outputs.arrays.capacity == 0
    for n_points, pairs in ((1000, 80000), (10, 800), (3000, 240000)):
        outputs.allocate_guess((80000, 1000), n_points)
        assert pairs <= outputs.arrays.capacity <= pairs + pairs // 8 + 256


def test_room_that_is_not_there(monkeypatch):
    """A guess that does not fit is no error: the engine asks for what it needs."""
    empty = torch.empty
    outputs = _outputs_of()
    full = [True]

    def no_room_for_vectors(shape, **options):
        if full and isinstance(shape, tuple) and options["dtype"] == torch.float64:
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(shape, **options)

    monkeypatch.setattr(torch, "empty", no_room_for_vectors)
    outputs.allocate_guess((760, 10), 10)
    arrays = outputs.arrays
    assert arrays.capacity == 0 and not any((arrays.i, arrays.j, arrays.pairs, arrays.shifts, arrays.distances, arrays.vectors))
    assert outputs.i is None and outputs.shifts is None
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device: _Stream(0, []))
    full.clear()
    with outputs:
        assert _outputs.allocate_callback(None, 700, ctypes.byref(outputs.arrays)) == 0
        assert outputs.arrays.capacity == 700
        # one that the engine asks for is the caller's error
        full.append(True)
        assert _outputs.allocate_callback(None, 1000, ctypes.byref(outputs.arrays)) == 1
    assert isinstance(outputs.error, torch.cuda.OutOfMemoryError)


@pytest.mark.parametrize("n_pairs", [0, 1, 60, 128, 700, 100000])
@pytest.mark.parametrize("capacity", [1.0, 1.06, 1.12, 1.2, 4.0])
def test_storage_of_a_list(n_pairs, capacity):
    """A list that is kept or saved takes little more than its own rows with it."""
    outputs = _outputs_of()
    outputs.allocate(int(n_pairs * capacity) + 64)
    for tensor in outputs.take(n_pairs):
        assert len(tensor) == n_pairs
        row = tensor.element_size() * (3 if tensor.dim() == 2 else 1)
        assert tensor.untyped_storage().nbytes() <= row * (n_pairs + n_pairs // 8 + 128)
