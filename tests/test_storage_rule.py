"""Which wavefield storage the default ``grad_mode="checkpoint"`` takes: the whole history while such histories take no
more than an eighth of the memory budget, those already alive included, else checkpoints of ``ceil(sqrt(n_steps))``
steps; the gradient is bitwise the same either way."""

from __future__ import annotations

import math

import pytest
import torch

from conftest import cotangent, load_golden
from nefi_b200.plan import plan_storage
from test_gpu_parity import make_op


class Plan:
    pml = None

    def level_bytes(self, n_shots):
        return 1000 * n_shots

    def snapshot_bytes(self, n_shots, n_snap, kind):
        return 2000 * n_shots * n_snap


def test_an_eighth_of_the_budget_is_the_line():
    n, hist = 100, (100 + 3) * 1000

    def mode(budget, **kw):
        return plan_storage(Plan(), 1, n, "checkpoint", kw.pop("every", None), kw.pop("snapshot", "exact"), budget, **kw)

    assert mode(8 * hist) == ("history", None)
    assert mode(8 * hist - 1) == ("checkpoint", 10)
    assert mode(16 * hist, held=hist) == ("history", None)
    assert mode(16 * hist - 1, held=hist) == ("checkpoint", 10)
    assert mode(None) == ("checkpoint", 10)  # no budget known
    assert mode(80 * hist, every=7) == ("checkpoint", 7)
    assert mode(80 * hist, snapshot="delta16") == ("checkpoint", 10)
    assert mode(80 * hist, checkpoint_slots=3) == ("checkpoint", 10, 3)


def _hist(op, device, dtype, shots):
    return (op.n_steps + 3) * op._plan(device, dtype).level_bytes(shots)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("name", ["fwi_o4_sponge", "fwi_o4_cerjan", "fwi_o4_pml", "fwi_o2_pml_aniso", "pat3d_o2_sponge"])
def test_default_checkpoints_give_the_gradient_of_the_history(name, dtype, cuda_device):
    """On both sides of the line, at the default segment length."""
    case = load_golden(name)
    got = []
    for eighths in (8, 7):
        op = make_op(case, grad_mode="checkpoint")
        if case["kind"] == "fwi":
            op.memory_budget = eighths * _hist(op, cuda_device, dtype, op.n_sources)
            x = [torch.tensor(case["c"], dtype=dtype, device=cuda_device, requires_grad=True)]
            tr = op({"c": x[0]})
        else:
            x = [torch.tensor(case[k], dtype=dtype, device=cuda_device, requires_grad=True) for k in ("p0", "c")]
            op.memory_budget = eighths * _hist(op, cuda_device, dtype, max(1, x[0].numel() // x[1].numel()))
            tr = op.with_speed(*x)
        fn = tr.grad_fn
        while not hasattr(fn, "run"):
            fn = fn.next_functions[0][0]
        kind, every = ("history", None) if eighths == 8 else ("checkpoint", math.ceil(math.sqrt(op.n_steps)))
        assert fn.run.kind == kind and fn.run.storage.segment == (every or 0)
        g = torch.tensor(cotangent(tr.shape, 3), dtype=dtype, device=cuda_device)
        got.append((tr.detach(), *torch.autograd.grad((tr * g).sum(), x)))
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.gpu
def test_histories_alive_count_against_the_eighth(cuda_device):
    """Source chunks whose graphs are all alive until backward, and gradient graphs, together keep an eighth."""
    case = load_golden("fwi_o4_sponge")
    op = make_op(case, grad_mode="checkpoint")
    op.sources = op.sources[:1].repeat(5, 1) + torch.linspace(0, 0.01, 5, dtype=torch.float64)[:, None]
    op.source_batch = 1
    op.memory_budget = 20 * _hist(op, cuda_device, torch.float32, 1)
    c = torch.tensor(case["c"], dtype=torch.float32, device=cuda_device, requires_grad=True)
    for _ in range(2):  # the backward gives the histories back
        tr = op({"c": c})
        kinds = [f[0].run.kind for f in tr.grad_fn.next_functions]
        assert kinds == ["history"] * 2 + ["checkpoint"] * 3
        torch.autograd.grad(tr.sum(), c)
    obs = torch.zeros(tr.shape, device=cuda_device)
    op.source_batch, op.memory_budget = None, 9 * _hist(op, cuda_device, torch.float32, 5)
    first = op.gradient_graph(c.detach(), obs)
    assert op.last_storage == ("history", None)
    second = op.gradient_graph(c.detach(), obs)
    assert op.last_storage[0] == "checkpoint"
    assert torch.equal(first.run(c.detach(), obs)[1], second.run(c.detach(), obs)[1])
    first.release()
    del first
    op.gradient_graph(c.detach(), obs)
    assert op.last_storage == ("history", None)


@pytest.mark.gpu
def test_an_operators_own_budget_counts_its_own_histories(cuda_device):
    case = load_golden("fwi_o4_sponge")
    c = torch.tensor(case["c"], dtype=torch.float32, device=cuda_device, requires_grad=True)
    other = make_op(case)({"c": c})  # a history alive on the device
    op = make_op(case, grad_mode="checkpoint")
    op.memory_budget = 8 * _hist(op, cuda_device, torch.float32, op.n_sources)
    tr = op({"c": c})
    assert op.last_storage == ("history", None)
    op({"c": c})
    assert op.last_storage[0] == "checkpoint"
    del other, tr
