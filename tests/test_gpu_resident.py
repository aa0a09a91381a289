"""Sweeps of many steps per launch (resident2d.cuh) against the one-step launches.

``simulate(c, observe=...)`` advances one launch per step, ``simulate(c)`` and the operator take the whole
sweep in one launch when the grid fits; the arithmetic of a cell is the same, so fields are bitwise equal.
The grids put slab edges, strip remainders and partial vectors of columns at different places: one slab and
sixteen, strips of one to several heights, widths that are not a multiple of the vector.
"""

from __future__ import annotations

import pytest
import torch

from nefi_b200 import WaveOperatorB200
from nefi_b200._compat import Domain

pytestmark = pytest.mark.gpu

GRIDS = [(21, 34), (50, 47), (130, 61), (47, 331), (200, 203)]


def _op(shape, absorbing, order, receivers=None, **kw):
    n0, n1 = shape
    h = 10.0
    dom = Domain(shape, ((0.0, n0 * h), (0.0, n1 * h)))
    src = [[0.31 * n0 * h, 0.47 * n1 * h], [0.8 * n0 * h, 0.2 * n1 * h], [0.05 * n0 * h, 0.95 * n1 * h]]
    rec = receivers or [[(0.03 + 0.94 * i / 30) * n0 * h, (0.5 + 0.4 * (-1) ** i) * n1 * h] for i in range(31)]
    return WaveOperatorB200(dom, src, rec, n_t=17, dt_obs=1.7e-3, f0=25.0, c_max=2600.0, order=order,
                            absorbing=absorbing, absorb_width=7 * h, **kw)


def _speed(shape, dtype, device):
    x = torch.linspace(0, 1, shape[0], dtype=torch.float64)[:, None]
    z = torch.linspace(0, 1, shape[1], dtype=torch.float64)[None, :]
    return (2000.0 + 400.0 * z + 120.0 * torch.sin(9 * x + 4 * z)).to(dtype).to(device)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("absorbing", ["none", "sponge", "cerjan", "pml"])
@pytest.mark.parametrize("shape", GRIDS)
def test_resident_sweep_is_bitwise_the_one_step_launches(shape, absorbing, order, dtype, cuda_device):
    op = _op(shape, absorbing, order)
    c = _speed(shape, dtype, cuda_device)
    levels = []
    one, _ = op.simulate(c, observe=lambda st, n: levels.append(st[1].clone()), record=range(op.n_steps + 1))
    many, traces = op.simulate(c)
    assert float(one[1].abs().max()) > 0
    for a, b in zip(one, many):
        assert torch.equal(a, b)
    # the samples of the receivers from the one-step levels (the sampling's own rounding apart)
    corner, w = op.grid.point_stencils(op.receivers)
    idx = op.grid.flat_indices(corner).to(cuda_device)
    for j, tr in enumerate(traces):
        p = levels[j * op.substeps].flatten(1)
        ref = (p[:, idx].double() * w.to(cuda_device)).sum(-1)
        eps = torch.finfo(dtype).eps
        assert torch.allclose(tr.double(), ref, rtol=0, atol=8 * eps * float(p.abs().max()))


@pytest.mark.parametrize("absorbing", ["sponge", "pml"])
@pytest.mark.parametrize("line", ["rows", "columns", "coincident"])
def test_receivers_crowded_in_one_slab_match_the_oracle(absorbing, line, cuda_device):
    """Receivers that all lie in one slab, one per slab row and edge, or several on the same cell: traces and
    gradient in float64 against the float64 oracle."""
    import numpy as np
    import oracle

    from conftest import cotangent, rel_l2

    shape, h = (90, 76), 10.0
    rec = {"rows": [[445.0, 3.0 + 9.7 * i] for i in range(77)],
           "columns": [[5.0 + 9.9 * i, 401.0] for i in range(90)],
           "coincident": [[433.0, 288.0]] * 5 + [[434.0 + i, 288.0] for i in range(12)]}[line]
    op = _op(shape, absorbing, 4, rec, grad_mode="autograd")
    c = _speed(shape, torch.float64, cuda_device).requires_grad_(True)
    tr = op({"c": c})
    g = cotangent(tr.shape, 5)
    (gc,) = torch.autograd.grad((tr * torch.tensor(g, device=cuda_device)).sum(), c)
    orc = oracle.OracleWave(shape, tuple(tuple(e) for e in op.domain.extent), np.asarray(rec),
                            sources=op.sources.numpy(), n_t=17, dt_obs=1.7e-3, f0=25.0, c_max=2600.0, order=4,
                            absorbing=absorbing, absorb_width=7 * h)
    tr_o, gc_o = orc.fwi(c.detach().cpu().numpy(), g, dtype=np.float64)
    assert rel_l2(tr.detach().cpu().numpy(), tr_o) < 1e-11
    assert rel_l2(gc.cpu().numpy(), gc_o) < 1e-10
