"""The first resident sweep of a process inside a stream capture: what the library sets up once (the report words in pinned
host memory, cluster occupancies, kernel attributes) is set up there, and the replay gives the eager results."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys, torch
sys.path[:0] = [{root!r}, {tests!r}, {oracle!r}]
from test_gpu_resident import _op, _speed
from nefi_b200.operators import _forward_sweep, _Run
dev = torch.device("cuda", 0)
op, c = _op((90, 76), "sponge", 4), _speed((90, 76), torch.float32, dev)
plan = op._plan(dev, torch.float32)
c2dt2 = plan.empty_levels(1, 1)[0, 0]
run = _Run(plan, 3, op.n_steps, ("ring", None), "exact")
traces = torch.zeros(3, plan.n_rec, op.n_t, device=dev)
medium, acq = plan.medium(c2dt2), plan.acquisition(3)
import ctypes as C
from nefi_b200 import _lib
_lib.check(_lib.load().nw_prepare_medium(C.byref(plan.g), plan.n_abs, c.data_ptr(), op.dt**2, c2dt2.data_ptr(), 0))
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    run.ring.zero_()
    _forward_sweep(plan, medium, acq, run, 0, op.n_steps, traces, _lib.stream_handle(dev))
assert plan.sweep_route(3)[0] > 1
g.replay()
torch.cuda.synchronize()
_, eager = op.simulate(c)
assert float(traces.abs().max()) > 0 and torch.equal(traces, torch.stack(eager, -1))
assert _lib.load().nw_reported() == _lib.NW_OK
print("same")
"""


def test_first_sweep_of_a_process_is_captured(cuda_device):
    root = Path(__file__).resolve().parents[1]
    src = SCRIPT.format(root=str(root), tests=str(root / "tests"), oracle=str(root / "oracle"))
    out = subprocess.run([sys.executable, "-c", src], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "same", out.stderr[-2000:]
