"""A resident sweep in which a CTA's rows do not come (resident2d.cuh): the waits for them run out, the sweep ends, what it
wrote is NaN, the host is told once, and the device goes on working. ``NW_TUNE_MUTE`` keeps the first CTA of each shot
from sending."""

from __future__ import annotations

import pytest
import torch

from nefi_b200 import _lib
from nefi_b200.plan import ghost_view
from test_gpu_resident import _op, _speed

pytestmark = pytest.mark.gpu


def _set(op, flags):
    for plan in op._plans.values():
        plan.tuning.flags = flags


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("absorbing,order", [("none", 2), ("sponge", 4), ("pml", 2), ("pml", 4)])
@pytest.mark.parametrize("shape", [(50, 47), (130, 121)])
def test_rows_that_do_not_come_are_reported(shape, absorbing, order, dtype, cuda_device):
    lib = _lib.load()
    op = _op(shape, absorbing, order, grad_mode="autograd")
    c = _speed(shape, dtype, cuda_device).requires_grad_(True)
    tr = op({"c": c})
    (g,) = torch.autograd.grad(tr.sum(), c)
    plan = op._plan(cuda_device, dtype)
    assert plan.sweep_route(3)[0] > 1 and plan.sweep_route(3, adjoint=True)[0] > 1
    _set(op, _lib.MUTE)
    state, obs = op.simulate(c.detach())
    torch.cuda.synchronize()
    assert all(torch.isnan(p).all() for p in (*state, *obs))
    with pytest.raises(_lib.LibraryError, match="gave up") as e:  # the next call says so, once
        op.simulate(c.detach())
    assert e.value.code == _lib.NW_ERR_TIMEOUT
    assert lib.nw_reported() == _lib.NW_OK == lib.nw_status(_lib.stream_handle(cuda_device))
    lap = op({"c": c}).grad_fn.run  # a history of NaN
    torch.cuda.synchronize()
    assert lib.nw_reported() == _lib.NW_ERR_TIMEOUT
    assert all(torch.isnan(ghost_view(plan.g, f)).all() for f in lap.history.flatten(0, 1)[-3:])
    # the adjoint
    _set(op, 0)
    tr2 = op({"c": c})
    _set(op, _lib.MUTE)
    (bad,) = torch.autograd.grad(tr2.sum(), c)
    assert lib.nw_status(_lib.stream_handle(cuda_device)) == _lib.NW_ERR_TIMEOUT
    assert torch.isnan(bad).all() and lib.nw_reported() == _lib.NW_OK
    # and everything works as before
    _set(op, 0)
    tr3 = op({"c": c})
    (g3,) = torch.autograd.grad(tr3.sum(), c)
    assert torch.equal(tr3, tr) and torch.equal(g3, g)
    assert lib.nw_status(_lib.stream_handle(cuda_device)) == _lib.NW_OK


def test_a_gradient_graph_and_a_batch_report_it(cuda_device):
    from nefi_b200.batched import BatchedFWI

    shape = (200, 203)  # more than one CTA can hold, in a batch too
    op = _op(shape, "sponge", 4, grad_mode="checkpoint", checkpoint_every=8)
    c = _speed(shape, torch.float32, cuda_device)
    obs = torch.zeros(op.n_sources, op.n_receivers, op.n_t, device=cuda_device)
    g = op.gradient_graph(c, obs)
    want = g.run(c, obs)[1].clone()
    _set(op, _lib.MUTE)
    op.simulate(c)  # eager, on the same device
    torch.cuda.synchronize()
    with pytest.raises(_lib.LibraryError, match="gave up"):
        g.replay()
    _set(op, 0)
    assert torch.equal(g.run(c, obs)[1], want)
    bt = BatchedFWI([op], device=cuda_device, segment=8, snapshot="exact", tuning=(0, 0, 0, 0, 0, 0, 0, _lib.MUTE))
    with pytest.raises(_lib.LibraryError, match="gave up"):
        for _ in range(2):
            bt.misfit_gradients([c], [obs])
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    _lib.load().nw_reported()  # (the sweeps of the call that was told, if they were under way)
