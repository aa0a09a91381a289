"""nw_grid.core_lo / core_hi, by which the steps leave the layer's coefficients out: without a layer they mean nothing, with
one a box that reaches beyond the grid, or holds no cell, is no error (the coefficients are 1 where there is no layer)."""

from __future__ import annotations

import pytest
import torch

from nefi_b200 import _lib
from test_gpu_resident import _op, _speed

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, _lib.ONE_STEP_FORWARD | _lib.ONE_STEP_ADJOINT])
@pytest.mark.parametrize("absorbing,lo,hi", [("none", (-7, 3), (-5, -5)), ("none", (0, 0), (10**6, 10**6)),
                                             ("none", (40, 9), (12, 2)), ("sponge", (10**6, 0), (0, 0)),
                                             ("cerjan", (60, 50), (20, 10)), ("sponge", (0, 0), (0, 0))])
def test_any_core_box_gives_the_same_results(absorbing, lo, hi, flags, cuda_device):
    op = _op((66, 59), absorbing, 4, grad_mode="autograd")
    op.tuning = (0, 0, 0, 0, 0, 0, 0, flags)
    c = _speed((66, 59), torch.float32, cuda_device).requires_grad_(True)
    got = []
    for box in (None, (lo, hi)):
        plan = op._plan(cuda_device, torch.float32)
        if box:
            for ax in range(2):
                plan.g.core_lo[ax], plan.g.core_hi[ax] = box[0][ax], box[1][ax]
        assert (plan.sweep_route(3)[0] > 0) == (flags == 0)
        tr = op({"c": c})
        got.append((tr.detach(), torch.autograd.grad(tr.square().sum(), c)[0]))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert float(got[0][1].abs().max()) > 0
