"""What a new list costs beside its build: the runtime is asked for nothing but
the shared memory of the few kernels that take more than any kernel may."""

import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = """
import collections, json, torch, vesin_b200
from torch.profiler import ProfilerActivity, profile
points, box = torch.rand((48, 3), dtype=torch.float64, device="cuda"), torch.eye(3, dtype=torch.float64, device="cuda")
kept = vesin_b200.NeighborList(0.2, True)
kept.compute(points, box, False, "ijSdD")
torch.cuda.synchronize()
with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as calls:
    new = vesin_b200.NeighborList(0.2, True)
    new.compute(points, box, False, "ijSdD")
    torch.cuda.synchronize()
print(json.dumps(collections.Counter(event.name for event in calls.events())))
"""


def test_a_new_list_sets_up_few_kernels():
    done = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    calls = json.loads(done.stdout.splitlines()[-1])
    if not any(name.startswith("cudaLaunchKernel") for name in calls):
        pytest.skip("the calls of the runtime are not recorded here")
    assert calls.get("cudaFuncSetAttribute", 0) <= 8
