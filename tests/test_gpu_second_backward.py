"""A second backward through one photoacoustic call: refused where the first released the stored wavefield (the gradient
of the sound speed, or checkpoints asked for), the same gradient where nothing was stored."""

from __future__ import annotations

import pytest
import torch

from conftest import load_golden
from nefi_b200 import _lib
from nefi_b200._compat import OperatorError
from test_gpu_parity import make_op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["pat2d_o4_sponge", "pat3d_o2_sponge"])
def test_second_backward(name, cuda_device):
    case = load_golden(name)
    p0 = torch.tensor(case["p0"], device=cuda_device, requires_grad=True)
    c = torch.tensor(case["c"], device=cuda_device, requires_grad=True)
    for loss, x in ((make_op(case).with_speed(p0, c).square().sum(), (p0, c)),
                    (make_op(case, grad_mode="checkpoint", checkpoint_every=5)({"p0": p0}).square().sum(), (p0,))):
        torch.autograd.grad(loss, x, retain_graph=True)
        n0 = _lib.load().nw_launch_count()
        with pytest.raises(OperatorError, match="second backward"):
            torch.autograd.grad(loss, x)
        assert _lib.load().nw_launch_count() == n0
    loss = make_op(case)({"p0": p0}).square().sum()
    (g,) = torch.autograd.grad(loss, p0, retain_graph=True)
    assert torch.equal(torch.autograd.grad(loss, p0)[0], g) and float(g.abs().max()) > 0
