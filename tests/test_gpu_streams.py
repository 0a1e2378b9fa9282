"""Calculators called with work still queued on the caller's stream, the default
one and another: inputs that are being made, and (on the other stream) memory
for the outputs that was handed out a moment ago."""

import numpy as np
import pytest

from oracle import oracle as O
from vesin_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side_stream", [False, True])
@pytest.mark.parametrize("copy", [True, False])
@pytest.mark.parametrize("batch", [False, True])
def test_inputs_still_in_the_queue(side_stream, copy, batch):
    import torch

    import vesin_b200

    frames = [W.diamond(4, seed=s) for s in (1, 2)] + [W.diamond(5, seed=3)]
    device = torch.device("cuda", 0)
    on_device = [[torch.tensor(a, device=device) for a in frame[:2]] for frame in frames]
    calculator = (vesin_b200.BatchNeighborList if batch else vesin_b200.NeighborList)(5.0, True)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream() if side_stream else torch.cuda.default_stream()):
        for (points, box, _), (there, box_there) in zip(frames, on_device):
            expected = O.canonical(O.restated_neighbors(points, box, [not batch] * 3, 5.0, True, "ijSdD"))
            late = torch.zeros_like(there)
            torch.cuda._sleep(20_000_000)  # 10 ms or so
            late.copy_(there)
            if batch:
                outputs, _ = calculator.compute(late, [0, len(points)], quantities="ijSdD", copy=copy)
            else:
                outputs = calculator.compute(late, box_there, True, "ijSdD", copy=copy)
            got = {key: value.cpu().numpy() for key, value in zip("ijSdD", outputs)}
            for key in "ij":
                got[key] = got[key].astype(np.int64)
            got = O.canonical(got)
            for key in "ijSdD":
                assert np.array_equal(got[key], expected[key]), key


def test_outputs_are_allocated_before_the_wait(monkeypatch):
    """On another stream the engine is not ordered behind an allocation: every
    allocation of a call has a wait for the stream after it, before the engine
    writes (recorded around the calls, with and without a guess of the length)."""
    import torch

    import vesin_b200
    from vesin_b200 import _outputs

    events = []
    allocate, synchronize = _outputs.OutputTensors.allocate, torch.cuda.Stream.synchronize
    monkeypatch.setattr(_outputs.OutputTensors, "allocate", lambda self, n: (allocate(self, n), events.append("allocate"))[0])
    monkeypatch.setattr(torch.cuda.Stream, "synchronize", lambda self: (synchronize(self), events.append("wait"))[0])
    points, box, _ = W.diamond(3)
    points, box = torch.tensor(points, device="cuda"), torch.tensor(box, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        for compute in (
            lambda c=vesin_b200.NeighborList(5.0, True): c.compute(points, box, True, "ijd"),
            lambda c=vesin_b200.BatchNeighborList(5.0, True): c.compute(points, [0, len(points)], quantities="ijd"),
        ):
            compute()
            assert events == ["wait", "allocate", "wait"]  # the engine asked for what the list needs
            events.clear()
            compute()
            assert events == ["allocate", "wait"]
            events.clear()
