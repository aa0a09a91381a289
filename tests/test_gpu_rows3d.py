"""The 3-D step on rows cut into parts (stencil3d.cuh: a tile holds at most 40 16-byte vectors of a row, so float32 rows
past 160 columns and float64 rows past 80 take two and more), with remainders of tiles in every axis, against the float64
oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import cotangent, rel_l2
from nefi_b200 import WaveInitialConditionOperatorB200
from nefi_b200._compat import Domain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tt,tg", [(torch.float32, 1e-5, 1e-4), (torch.float64, 1e-11, 1e-10)])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("shape,width", [((9, 11, 161), 0), ((7, 13, 173), 3), ((35, 6, 330), 2), ((12, 19, 83), 0)])
def test_rows_of_several_tiles(shape, width, order, dtype, tt, tg, cuda_device):
    import oracle

    h = 0.1
    extent = tuple((0.0, n * h) for n in shape)
    gen = torch.Generator().manual_seed(sum(shape) + order)
    p0 = torch.randn((2, *shape), generator=gen, dtype=torch.float64)
    c = 1.0 + 0.2 * torch.rand(shape, generator=gen, dtype=torch.float64)
    rec = [[(0.5 + 0.9 * (i % shape[0])) * h, 0.45 * shape[1] * h, (0.7 + 0.97 * i * (shape[2] - 2) / 40) * h] for i in range(40)]
    kw = dict(n_t=9, dt_obs=0.06, order=order, absorbing="sponge" if width else "none", absorb_width=width * h, c_max=1.25)
    op = WaveInitialConditionOperatorB200(Domain(shape, extent), rec, c=c, grad_mode="autograd", **kw)
    xs = [t.to(dtype).to(cuda_device).requires_grad_(True) for t in (p0, c)]
    tr = op.with_speed(*xs)
    g = cotangent(tr.shape, 7)
    gp, gc = torch.autograd.grad((tr * torch.tensor(g, dtype=dtype, device=cuda_device)).sum(), xs)
    orc = oracle.OracleWave(shape, extent, np.asarray(rec), **kw)
    otr, ogp, ogc = orc.pat(p0.numpy(), c.numpy(), g, dtype=np.float64)
    assert rel_l2(tr.detach().cpu().numpy(), otr) < tt
    assert rel_l2(gp.cpu().numpy(), ogp) < tg
    assert rel_l2(gc.cpu().numpy(), ogc) < tg
    # p0 alone: the adjoint without the velocity gradient
    (alone,) = torch.autograd.grad((op({"p0": xs[0]}) * torch.tensor(g, dtype=dtype, device=cuda_device)).sum(), xs[0])
    assert rel_l2(alone.cpu().numpy(), ogp) < tg
