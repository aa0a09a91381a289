"""The batched calls ignore a problem's schedule fields and ring levels (nw_storage), whichever way its sweeps run."""

from __future__ import annotations

import pytest
import torch

from nefi_b200 import _lib
from nefi_b200.batched import BatchedFWI
from test_gpu_batched import K, _batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, _lib.ONE_STEP_FORWARD | _lib.ONE_STEP_ADJOINT])
def test_schedule_fields_and_ring_levels_are_ignored(flags, cuda_device):
    ops, cs, obs = _batch(torch.float32, cuda_device)
    bt = BatchedFWI(ops, device=cuda_device, segment=K, snapshot="exact", tuning=(0, 0, 0, 0, 0, 0, 0, flags))
    _, grads = bt.misfit_gradients(cs, obs)
    want = [g.clone() for g in grads]
    none = torch.full((64,), -1, dtype=torch.int32)  # "no segment start goes into a slot"
    program = torch.zeros(3, dtype=torch.int32)
    for q, b in zip(bt.problems, bt.bufs):
        b["ring"] = b["plan"].empty_levels(4, b["S"])  # (room for what the field says)
        q.storage.ring, q.storage.ring_levels = b["ring"].data_ptr(), 4
        q.storage.snap_slot, q.storage.schedule, q.storage.n_schedule = none.data_ptr(), program.data_ptr(), 1
        b["snap"].zero_()
    _lib.check(_lib.load().nw_batch_prepare(bt.problems, len(ops), bt.tune, bt.table.data_ptr(),
                                            _lib.stream_handle(cuda_device)))
    _, grads = bt.misfit_gradients(cs, obs)
    assert all(torch.equal(a, b) for a, b in zip(grads, want)) and all(float(g.abs().max()) > 0 for g in want)
