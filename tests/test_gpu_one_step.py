"""The launches of one step (fwd2d, adj2d, the PML's layer launch and fork, the batch kernels), which large grids take.

The grids of the other GPU tests fit a resident sweep, so here those tests run again with every plan asking for one
step per launch (``nw_tuning.flags``), and the two ways are compared with each other.
"""

from __future__ import annotations

import pytest
import torch

from conftest import cotangent, load_golden, rel_l2
from nefi_b200 import WaveOperatorB200, _lib
from nefi_b200._compat import Domain
from nefi_b200.batched import BatchedFWI, autotune
from nefi_b200.plan import DevicePlan
from test_gpu_batched import (  # noqa: F401  (collected here, under the fixture below)
    _problem,
    test_batch_equals_each_problem_alone,
    test_fused_misfit_batch_equals_each_problem_alone_and_replays,
    test_graph_replay_equals_eager_batch,
    test_pml_batch_graph_replay_equals_eager,
    test_pml_problems_in_a_batch_equal_each_problem_alone,
)
from test_gpu_graph import test_graph_replay_is_bitwise_misfit_gradient  # noqa: F401
from test_gpu_parity import (  # noqa: F401
    _layered_grad,
    _layered_op,
    make_op,
    test_binomial_checkpointing_is_identical_to_full_history,
    test_checkpointed_16_bit_gradient_of_a_salt_model_meets_the_budget,
    test_checkpointed_gradient_is_identical_to_full_history,
    test_fwi_float32_matches_reference_float32,
    test_fwi_float64_matches_reference,
    test_multiresolution_source_batching_and_speed_check,
    test_pat_adjoint_identity_and_linearity_float64,
    test_pat_float64_matches_reference,
    test_pml_cotangents_of_layer_cells_match_the_oracle,
    test_pml_forward_captured_in_a_fresh_thread,
    test_pml_interior_through_tiled_kernels_matches_the_oracle,
    test_random_geometries_match_the_oracle_and_the_reference,
    test_results_do_not_depend_on_the_launch_shape,
    test_two_steps_per_launch_are_bitwise_one_step,
)
from test_gpu_time_reversal import (  # noqa: F401
    test_adjoint_time_reversal_is_the_operator_adjoint,
    test_coincident_receivers_keep_the_last_trace,
    test_dirichlet_time_reversal_matches_reference,
)

pytestmark = pytest.mark.gpu

ONE_STEP = _lib.ONE_STEP_FORWARD | _lib.ONE_STEP_ADJOINT


@pytest.fixture(autouse=True)
def one_step(request, monkeypatch):
    """Every plan asks for one step per launch, except in the tests below, which choose for themselves."""
    if request.function.__module__ == __name__:
        return
    set_tuning = DevicePlan.set_tuning

    def forced(self, *args, **kw):
        set_tuning(self, *args, **kw)
        self.tuning.flags = ONE_STEP
        assert self.sweep_route(1) == self.sweep_route(1, adjoint=True) == (0, 0)

    monkeypatch.setattr(DevicePlan, "set_tuning", forced)


def _gradient(op, c, g, flags):
    op.tuning = (0, 0, 0, 0, 0, 0, 0, flags)
    op._plans.clear()
    c = c.clone().requires_grad_(True)
    n0 = _lib.load().nw_launch_count()
    tr = op({"c": c})
    (gc,) = torch.autograd.grad((tr * g).sum(), c)
    return tr.detach(), gc, int(_lib.load().nw_launch_count() - n0)


def _both_ways(shape, shots, absorbing, order, dtype, dev, width=8):
    """A resident gradient against that of one-step launches: traces bitwise, the gradient up to the order of its sums
    (the tolerances of the launch-shape test). Returns the rows a thread steps, forward and adjoint."""
    h = 10.0
    n0, n1 = shape
    src = [[(k + 0.4) * n0 * h / shots, (0.2 + 0.6 * k / shots) * n1 * h] for k in range(shots)]
    rec = [[(i + 0.5) * h, (0.2 + 0.6 * (i * shots // n0) / shots) * n1 * h + (-1) ** i * 1.3 * h] for i in range(n0)]
    op = WaveOperatorB200(Domain(shape, ((0.0, n0 * h), (0.0, n1 * h))), src, rec, n_t=24, dt_obs=2.2e-3, f0=60.0,
                          c_max=2600.0, order=order, absorbing=absorbing, absorb_width=width * h, grad_mode="autograd")
    x = torch.linspace(0, 1, n0, dtype=torch.float64)[:, None]
    z = torch.linspace(0, 1, n1, dtype=torch.float64)[None, :]
    c = (2000.0 + 400.0 * z + 120.0 * torch.sin(9 * x + 4 * z)).to(dtype).to(dev)
    g = torch.tensor(cotangent((shots, len(rec), 24), 3), dtype=dtype, device=dev)
    tr0, g0, n_one = _gradient(op, c, g, ONE_STEP)
    assert n_one >= 2 * op.n_steps
    tr1, g1, n_many = _gradient(op, c, g, 0)
    plan = op._plan(dev, dtype)
    fwd, adj = plan.sweep_route(shots), plan.sweep_route(shots, adjoint=True)
    assert fwd[0] > 0 or adj[0] > 0
    assert n_many < 20 + op.n_steps * ((fwd[0] == 0) + (adj[0] == 0)) * (2 if absorbing == "pml" else 1)
    loud = float(tr0.abs().max())
    same = torch.equal(tr0, tr1)
    assert same and loud > 0
    assert rel_l2(g1.cpu().numpy(), g0.cpu().numpy()) < (1e-12 if dtype == torch.float64 else 1e-5)
    return fwd[1], adj[1]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("absorbing", ["none", "sponge", "cerjan", "pml"])
@pytest.mark.parametrize("shape,shots", [((50, 47), 3), ((130, 61), 5), ((203, 200), 6)])
def test_resident_gradient_is_that_of_one_step_launches(shape, shots, absorbing, order, dtype, cuda_device):
    rows = _both_ways(shape, shots, absorbing, order, dtype, cuda_device)
    assert all(rows) or shape[0] > 200


# (layer, cells a side, shots, dtype, rows a thread steps forward and adjoint at order 4; 0: not looked at here)
TALL = [("none", 200, 16, torch.float32, 6, 6), ("none", 256, 16, torch.float32, 8, 8),
        ("sponge", 256, 16, torch.float32, 12, 12), ("sponge", 400, 16, torch.float32, 12, 0),
        ("sponge", 200, 1, torch.float64, 6, 0), ("sponge", 168, 1, torch.float64, 0, 6),
        ("sponge", 128, 16, torch.float64, 8, 8), ("sponge", 168, 16, torch.float64, 12, 12),
        ("pml", 168, 16, torch.float32, 6, 0), ("pml", 256, 1, torch.float32, 6, 6),
        ("pml", 100, 16, torch.float64, 6, 0), ("pml", 168, 1, torch.float64, 0, 6)]


@pytest.mark.parametrize("order", [2, 4])
@pytest.mark.parametrize("absorbing,n,shots,dtype,fwd,adj", TALL)
def test_tall_strips(absorbing, n, shots, dtype, fwd, adj, order, cuda_device):
    """Strips of six rows a thread and more (twelve: the adjoint streams c^2 dt^2), as grids of 300^2 and up take."""
    rows = _both_ways((n, n), shots, absorbing, order, dtype, cuda_device, width=20)
    if order == 4:
        assert all(w in (0, r) for w, r in zip((fwd, adj), rows)), rows


@pytest.mark.parametrize("absorbing", ["sponge", "pml"])
def test_batch_of_resident_and_tiled_problems(absorbing, cuda_device):
    """A batch with problems of both kinds, whose resident members run on lanes beside the common launches: each
    gets what it gets alone, eager and replayed."""
    ops, cs, obs = [], [], []
    for n, shots, n_t, seed in [(40, 2, 31, 0), (632, 9, 24, 1), (64, 3, 45, 2), (33, 1, 20, 3), (616, 8, 28, 4)]:
        op, c = _problem(n, shots, n_t, seed, absorbing=absorbing)
        ops.append(op)
        cs.append(c.float().to(cuda_device))
        with torch.no_grad():
            obs.append(op({"c": cs[-1] * 0.97}))
    route = [[op._plan(cuda_device, torch.float32).sweep_route(op.n_sources, adj)[0] for adj in (False, True)] for op in ops]
    assert route[1] == route[4] == [0, 0] and all(f > 0 and a > 0 for f, a in (route[0], route[2], route[3]))
    bt = BatchedFWI(ops, device=cuda_device, segment=16, snapshot="exact")
    losses, grads = bt.misfit_gradients(cs, obs)
    losses, grads = [float(v) for v in losses], [g.clone() for g in grads]
    for i, op in enumerate(ops):
        loss, g = op.misfit_gradient(cs[i], obs[i])
        assert losses[i] == float(loss) and torch.equal(grads[i], g), i
        assert float(g.abs().max()) > 0
    bt.capture()
    _, again = bt.misfit_gradients(cs, obs)
    assert all(torch.equal(a, b) for a, b in zip(again, grads))


def test_a_flag_that_is_none_counts_as_no_flag(cuda_device):
    plan = make_op(load_golden("fwi_o4_sponge"))._plan(cuda_device, torch.float32)
    want = plan.sweep_route(2), plan.sweep_route(2, adjoint=True)
    assert want[0][0] > 0 and want[1][0] > 0
    for flags in (-1, 8, 0x7fffffff):
        plan.set_tuning(flags=flags)
        assert (plan.sweep_route(2), plan.sweep_route(2, adjoint=True)) == want
    plan.set_tuning(flags=_lib.ONE_STEP_ADJOINT)
    assert plan.sweep_route(2) == want[0] and plan.sweep_route(2, adjoint=True) == (0, 0)


def test_the_autotuners_time_only_what_can_be_chosen(cuda_device):
    """A direction whose sweep takes all its steps in one launch runs the same kernel under every shape."""
    op = _layered_op(shots=4, n_t=21)
    c = torch.full(op.domain.shape, 2400.0, device=cuda_device)
    plan = op._plan(cuda_device, torch.float32)
    assert plan.sweep_route(4)[0] and plan.sweep_route(4, adjoint=True)[0]
    tu = op.autotune(c, steps=20, repeats=1)
    assert {k[:3] for k in op.autotune_results if k[6] == 1} == {op.FWD_CANDIDATES[0][:3]}
    assert {k[3:6] for k in op.autotune_results} == {(0, 0, 0), op.ADJ_CANDIDATES[0]} and len(tu) == 7
    op64 = _layered_op(shots=4, n_t=21)  # (float64 takes no tile of four columns a thread)
    assert op64.autotune(c.double(), steps=20, repeats=1)[0] == 2
    large = _layered_op(n=600, shots=9, n_t=11)
    large.autotune(torch.full(large.domain.shape, 2400.0, device=cuda_device), steps=10, repeats=1)
    assert len(large.autotune_results) >= len(op.FWD_CANDIDATES) + len(op.ADJ_CANDIDATES)
    small = [_problem(n, 2, 31, n)[0] for n in (40, 56)]
    tuning, times = autotune(small, steps=20, device=cuda_device, repeats=1)
    assert len(times) == 2 and all(v > 0 for v in tuning)
    mixed = small + [_problem(632, 9, 24, 1)[0]]
    assert len(autotune(mixed, steps=20, device=cuda_device, repeats=1)[1]) == 10
