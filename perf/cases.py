"""Performance cases: what a user of the wave operators has them do, over the range of sizes in use.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare``/``run`` build and
execute one pass through the public entry points, ``work`` counts the bytes and operations a pass cannot
do without, and ``exact`` evaluates the same pass in plain float64 torch.

Kinds of case:

* ``fwi``: acoustic full-waveform inversion on a 2-D grid. ``forward`` returns the traces; ``gradient`` runs
  the operator, the least-squares misfit and ``backward()`` as a solver does, and returns traces and gradient;
  ``graph`` replays a recorded gradient, as a long inversion does.
* ``batch``: independent FWI problems of uneven size advanced together, from one recorded graph.
* ``pat``: photoacoustic tomography on a 3-D grid: traces of an initial pressure and its gradient.
* ``reversal``: the time-reversal reconstruction of a 2-D initial pressure from receiver traces.
* ``misfit``: the band-limited trace misfit with the sensors' response, and its adjoint source.
"""

from __future__ import annotations

import math

import torch

from nefi_b200 import WaveInitialConditionOperatorB200, WaveOperatorB200, time_reversal
from nefi_b200._compat import Domain
from nefi_b200.batched import BatchedFWI
from nefi_b200.misfit import TraceMisfit

C_MAX = 4500.0  # m/s, the bound of the FWI models' speeds
DEV = "cuda"


def _fwi(name, n0, n1, shots, recs, steps, absorbing, call, **kw):
    return {"name": name, "kind": "fwi", "n0": n0, "n1": n1, "shots": shots, "recs": recs, "steps": steps,
            "substeps": 1, "absorbing": absorbing, "layer": 20, "order": 4, "dtype": "float32", "call": call,
            "storage": "autograd", "snapshot": "exact", **kw}


def listed():
    return [
        # the smallest useful call: one shot of a 128^2 line, traces only (data of a trial model)
        _fwi("fwi_128_forward", 128, 128, 1, 128, 1000, "sponge", "forward"),
        # a laptop-sized inversion with every option at its default: PML of 10 cells, checkpointed gradient,
        # odd extents, two leapfrog steps per trace sample
        _fwi("fwi_default_small", 97, 121, 5, 61, 400, "pml", "gradient", storage="checkpoint", layer=10, substeps=2),
        # the inner loop of a long inversion: a recorded gradient replayed on new models
        _fwi("fwi_256_graph", 256, 256, 4, 256, 500, "sponge", "graph"),
        # the benchmark grid: 16 shots, the whole history in device memory
        _fwi("fwi_512_sponge", 512, 512, 16, 512, 800, "sponge", "gradient"),
        # the same grid with the default layer and the default (checkpointed) gradient
        _fwi("fwi_512_pml", 512, 512, 16, 512, 400, "pml", "gradient", storage="checkpoint"),
        # a float64 gradient (a check against finite differences) on a ragged grid, Cerjan layer, order 2
        _fwi("fwi_cerjan_f64", 301, 437, 5, 173, 300, "cerjan", "gradient", order=2, dtype="float64", layer=13),
        # the large model: checkpointed with 16-bit snapshots
        _fwi("fwi_2048_ckpt16", 2048, 2048, 8, 2048, 120, "sponge", "gradient", storage="checkpoint",
             snapshot="delta16"),
        # data generation: float64 traces from the model on a grid refined two times
        _fwi("datagen_1024_f64", 1024, 1024, 16, 512, 200, "sponge", "forward", dtype="float64", layer=40),
        # uneven problems of one survey campaign advanced together
        {"name": "fwi_batch_uneven", "kind": "batch", "problems": 10, "steps": 300, "scale": 1.0},
        # a photoacoustic volume: traces on a sensor plane and the gradient of the initial pressure
        {"name": "pat_256", "kind": "pat", "n": 256, "batch": 2, "sensors": 256, "steps": 36, "order": 2,
         "storage": "checkpoint"},
        # the classical reconstruction on a 2-D slice, with the default layer
        {"name": "reversal_256", "kind": "reversal", "n0": 256, "n1": 250, "recs": 128, "steps": 600},
        # the misfit of a whole survey: sensor response, low-pass, muted traces, relative
        {"name": "misfit_survey", "kind": "misfit", "shots": 16, "recs": 512, "n_t": 4001, "dtype": "float32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fwi"] * 7 + ["batch", "pat", "reversal", "misfit"])
    if kind == "batch":
        return {"kind": "batch", "problems": rng.randint(3, 10), "steps": _log(rng, 60, 300),
                "scale": round(rng.uniform(0.25, 1.0), 3)}
    if kind == "pat":
        n = _log(rng, 40, 220)
        return {"kind": "pat", "n": n, "batch": rng.randint(1, 3 if n < 160 else 2), "sensors": max(8, n // rng.randint(1, 4)),
                "steps": _log(rng, 20, 48), "order": rng.choice([2, 2, 4]), "storage": rng.choice(["checkpoint", "autograd"])}
    if kind == "reversal":
        return {"kind": "reversal", "n0": _log(rng, 60, 500), "n1": _log(rng, 60, 500), "recs": _log(rng, 16, 512),
                "steps": _log(rng, 100, 600)}
    if kind == "misfit":
        return {"kind": "misfit", "shots": rng.randint(1, 16), "recs": _log(rng, 16, 512), "n_t": _log(rng, 150, 4001),
                "dtype": rng.choice(["float32", "float32", "float64"])}
    n0, n1, shots = _log(rng, 60, 1400), _log(rng, 60, 1400), rng.randint(1, 20)
    most = max(40, int(2.4e9 / (n0 * n1 * shots)))  # cell updates of a sweep, below the listed gradients'
    case = _fwi("", n0, n1, shots, _log(rng, 16, 900), _log(rng, 40, max(41, min(900, most))),
                rng.choice(["pml", "pml", "sponge", "sponge", "cerjan", "none"]),
                rng.choice(["gradient", "gradient", "gradient", "forward", "graph"]),
                storage=rng.choice(["checkpoint", "autograd"]), snapshot=rng.choice(["exact", "exact", "delta16"]),
                layer=rng.randint(8, 30), substeps=rng.choice([1, 1, 2]), order=rng.choice([4, 4, 2]),
                dtype=rng.choice(["float32", "float32", "float32", "float64"]))
    if case["dtype"] == "float64":
        case["snapshot"] = "exact"
    del case["name"]
    return case


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
H, F0 = 10.0, 10.0  # FWI: cell size (m) and Ricker peak frequency (Hz)


def _dt_obs(case):
    """Sampling interval: 0.4 h / c_max per leapfrog step."""
    return 0.4 * H / C_MAX * case["substeps"]


def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * (seed % 1000003) + salt)


def _layered(n0, n1, seed, salt=0):
    """Speeds (float64, n0 x n1): layers dipping along the second axis (depth) with smooth anomalies."""
    g = _gen(seed, salt)
    u = torch.rand(32, generator=g, device=DEV, dtype=torch.float64)
    x = (torch.arange(n0, device=DEV, dtype=torch.float64) + 0.5)[:, None] / n0
    z = (torch.arange(n1, device=DEV, dtype=torch.float64) + 0.5)[None, :] / n1
    c = torch.full((n0, n1), 1600.0, device=DEV, dtype=torch.float64)
    for k in range(6):
        depth = 0.1 + 0.8 * (k + u[k]) / 6 + 0.1 * (u[6 + k] - 0.5) * (x - 0.5)
        c = c + 380.0 * (0.6 + 0.4 * u[12 + k]) * 0.5 * (1.0 + torch.tanh((z - depth) * n1 / 1.5))
    for k in range(4):
        r2 = (x - 0.2 - 0.6 * u[18 + k]) ** 2 * (n0 / n1) ** 2 + (z - 0.2 - 0.6 * u[22 + k]) ** 2
        c = c + (400.0 * u[26 + k] - 200.0) * torch.exp(-r2 / (2 * 0.06**2))
    return c.clamp(1500.0, 4400.0)


def _line(n0, count, depth, shift):
    """Points (count, 2) evenly along the first axis at a depth in cells, off the cell centres."""
    x = (torch.arange(count, dtype=torch.float64) + 0.5 + 0.3 * (shift - 0.5)) * n0 * H / count
    x = x.clamp(0.5 * H, (n0 - 0.5) * H)  # inside the cell centres, also without a layer around the grid
    return torch.stack([x, torch.full_like(x, depth * H)], 1)


def _arrivals(src, rec, n_t, dt, f0, speed, seed, dtype, scale):
    """Observed traces: Ricker arrivals along straight rays with noise of 2 %."""
    d = torch.cdist(src, rec).to(DEV)[..., None]
    t = torch.arange(n_t, device=DEV, dtype=torch.float64) * dt
    a2 = (math.pi * f0 * (t - 1.2 / f0 - d / speed)) ** 2
    w = (1.0 - 2.0 * a2) * torch.exp(-a2) / torch.sqrt(1.0 + d / d.max().clamp_min(1e-9) * 10)
    w = w + 0.02 * torch.randn(w.shape, generator=_gen(seed, 7), device=DEV, dtype=torch.float64)
    return (scale * w).to(dtype).contiguous()


def _problem(case, seed, salt=0):
    """One FWI problem's model, acquisition and data, as plain tensors."""
    n0, n1 = case["n0"], case["n1"]
    dtype = getattr(torch, case["dtype"])
    shift = float(torch.rand(1, generator=_gen(seed, salt + 3), device=DEV))
    src, rec = _line(n0, case["shots"], 1.5, shift), _line(n0, case["recs"], 2.5, shift)
    n_t = case["steps"] // case["substeps"] + 1
    c = _layered(n0, n1, seed, salt).to(dtype)
    obs = _arrivals(src, rec, n_t, _dt_obs(case), F0, 2000.0, seed + salt, dtype, 2e-9)
    return c, src, rec, n_t, obs


def _operator(case, src, rec, n_t):
    n0, n1 = case["n0"], case["n1"]
    domain = Domain((n0, n1), ((0.0, n0 * H), (0.0, n1 * H)), axes=("x", "z"))
    return WaveOperatorB200(domain, src, rec, n_t=n_t, dt_obs=_dt_obs(case), f0=F0, c_max=C_MAX, order=case["order"],
                            absorbing=case["absorbing"], absorb_width=case["layer"] * H, courant=0.9,
                            grad_mode=case["storage"], snapshot=case["snapshot"])


def _members(case, seed):
    """The batch's problems: grids of 256 to 768 cells a side, 4 to 16 shots, uneven step counts."""
    u = torch.rand(case["problems"], 3, generator=torch.Generator().manual_seed(17), dtype=torch.float64)
    out = []
    for k, (a, b, d) in enumerate(u.tolist()):
        n = int((256, 384, 512, 768)[k % 4] * case["scale"])
        out.append(_fwi("", n, n - int(30 * a), 4 + int(12.99 * b), n, int(case["steps"] * (0.4 + 0.6 * d)), "sponge",
                        "gradient", storage="checkpoint", snapshot="delta16"))
    return out


PAT_H, PAT_C = 1e-4, 1500.0


def _pat_inputs(case, seed):
    """Speed map, initial pressures (smooth-edged balls) and sensor plane of a photoacoustic volume."""
    n, b = case["n"], case["batch"]
    u = torch.rand(6 + b * 60, generator=_gen(seed, 5), device=DEV, dtype=torch.float64).tolist()
    x = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n
    X, Y, Z = x[:, None, None], x[None, :, None], x[None, None, :]
    c = PAT_C * (1.0 + 0.05 * torch.sin(2 * math.pi * ((1 + u[0]) * X + u[1])) * torch.sin(2 * math.pi * ((1 + u[2]) * Y + u[3]))
                 * torch.sin(2 * math.pi * ((1 + u[4]) * Z + u[5])))
    p0 = torch.zeros(b, n, n, n, device=DEV, dtype=torch.float32)
    for i in range(b):
        for k in range(12):
            v = u[6 + 60 * i + 5 * k:]
            r = torch.sqrt((X - 0.15 - 0.7 * v[0]) ** 2 + (Y - 0.15 - 0.7 * v[1]) ** 2 + (Z - 0.15 - 0.7 * v[2]) ** 2)
            p0[i] = torch.maximum(p0[i], ((0.2 + 0.8 * v[3]) * torch.sigmoid((0.03 + 0.06 * v[4] - r) * n)).float())
    m = case["sensors"]
    s = (torch.arange(m, dtype=torch.float64) + 0.5) * n * PAT_H / m
    SX, SY = torch.meshgrid(s, s, indexing="ij")
    sensors = torch.stack([SX.ravel(), SY.ravel(), torch.full((m * m,), 0.7 * PAT_H, dtype=torch.float64)], 1)
    dt = 0.3 * PAT_H / (1.05 * PAT_C)
    obs = 0.05 * torch.randn(b, m * m, case["steps"] + 1, generator=_gen(seed, 6), device=DEV, dtype=torch.float32)
    return c, p0, sensors, dt, obs


def _reversal_inputs(case, seed):
    n0, n1 = case["n0"], case["n1"]
    dt = 0.4 * PAT_H / PAT_C
    ang = torch.arange(case["recs"], dtype=torch.float64) * (2 * math.pi / case["recs"])
    # a ring of sensors, its centre off the cell faces (a receiver holds the cell that contains it)
    rec = torch.stack([0.5 * n0 + 0.313 + 0.45 * n0 * torch.cos(ang), 0.5 * n1 + 0.187 + 0.45 * n1 * torch.sin(ang)], 1) * PAT_H
    u = torch.rand(8, 2, generator=_gen(seed, 9), device=DEV, dtype=torch.float64).cpu()
    src = (0.25 + 0.5 * u) * torch.tensor([n0, n1], dtype=torch.float64) * PAT_H
    tr = _arrivals(src, rec, case["steps"] + 1, dt, 0.04 / dt, PAT_C, seed, torch.float32, 1.0).sum(0).contiguous()
    return rec, dt, tr


MISFIT_DT, MISFIT_FMAX, MISFIT_SENSOR, MISFIT_TAPER = 1e-3, 60.0, 90.0, 0.3


def _misfit_inputs(case, seed):
    dtype = getattr(torch, case["dtype"])
    shape = (case["shots"], case["recs"], case["n_t"])
    src, rec = _line(600, case["shots"], 1.5, 0.4), _line(600, case["recs"], 2.5, 0.4)
    f0 = min(25.0, 0.3 * case["n_t"])
    obs = _arrivals(src, rec, case["n_t"], MISFIT_DT, f0, 2000.0, seed, dtype, 1.0)
    pred = _arrivals(src, rec, case["n_t"], MISFIT_DT, f0, 2100.0, seed + 1, dtype, 1.1)
    mask = (torch.rand(*shape[:2], 1, generator=_gen(seed, 8), device=DEV) > 0.05).to(dtype)
    mask[0, 0] = 1
    return pred, obs, mask


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "fwi":
        c, src, rec, n_t, obs = _problem(case, seed)
        op = _operator(case, src, rec, n_t)
        st = {"kind": case["call"], "op": op, "c": c, "obs": obs}
        if case["call"] == "graph":
            st["graph"] = op.gradient_graph(c, obs)
        return st
    if kind == "batch":
        members = _members(case, seed)
        probs = [_problem(m, seed, 100 * k) for k, m in enumerate(members)]
        ops = [_operator(m, p[1], p[2], p[3]) for m, p in zip(members, probs)]
        batch = BatchedFWI(ops, snapshot="delta16")
        cs, obs = [p[0] for p in probs], [p[4] for p in probs]
        batch.misfit_gradients(cs, obs)
        batch.capture()
        return {"kind": kind, "batch": batch, "c": cs, "obs": obs}
    if kind == "pat":
        c, p0, sensors, dt, obs = _pat_inputs(case, seed)
        n = case["n"]
        domain = Domain((n, n, n), ((0.0, n * PAT_H),) * 3, axes=("x", "y", "z"))
        op = WaveInitialConditionOperatorB200(domain, sensors, n_t=case["steps"] + 1, dt_obs=dt, c=c.cpu(),
                                              order=case["order"], absorbing="sponge", absorb_width=16 * PAT_H,
                                              courant=0.9, grad_mode=case["storage"])
        return {"kind": kind, "op": op, "p0": p0, "obs": obs}
    if kind == "reversal":
        rec, dt, tr = _reversal_inputs(case, seed)
        n0, n1 = case["n0"], case["n1"]
        domain = Domain((n0, n1), ((0.0, n0 * PAT_H), (0.0, n1 * PAT_H)), axes=("x", "z"))
        return {"kind": kind, "domain": domain, "rec": rec, "dt": dt, "traces": tr}
    pred, obs, mask = _misfit_inputs(case, seed)
    mf = TraceMisfit(MISFIT_DT, MISFIT_FMAX, MISFIT_TAPER, True, MISFIT_SENSOR)
    return {"kind": kind, "misfit": mf, "pred": pred, "obs": obs, "mask": mask}


def run(st):
    kind = st["kind"]
    if kind == "forward":
        with torch.no_grad():
            return st["op"]({"c": st["c"]})
    if kind == "gradient":
        c = st["c"].detach().requires_grad_(True)
        traces = st["op"]({"c": c})
        (0.5 * (traces - st["obs"]).square().sum()).backward()
        return {"traces": traces.detach(), "grad": c.grad}
    if kind == "graph":  # the gradient in the model's type, as the model's update takes it
        loss, grad = st["graph"].run(st["c"], st["obs"])
        return {"loss": loss.clone(), "grad": grad.to(st["c"].dtype)}
    if kind == "batch":
        losses, grads = st["batch"].misfit_gradients(st["c"], st["obs"])
        return {"loss": [x.clone() for x in losses], "grad": [g.to(c.dtype) for g, c in zip(grads, st["c"])]}
    if kind == "pat":
        p0 = st["p0"].detach().requires_grad_(True)
        traces = st["op"]({"p0": p0})
        (0.5 * (traces - st["obs"]).square().sum()).backward()
        return {"traces": traces.detach(), "grad": p0.grad}
    if kind == "reversal":
        return time_reversal(st["traces"], st["domain"], st["rec"], dt_obs=st["dt"], c=PAT_C)
    st["misfit"].prepare(st["obs"], st["mask"], always=True)
    loss, grad = st["misfit"].value_and_grad(st["pred"])
    return {"loss": loss.clone(), "grad": grad}


# ------------------------------------------------------------------------------------------------
# work
# ------------------------------------------------------------------------------------------------
def _fwi_work(c):
    """A sweep reads and writes nothing but its inputs and outputs; its arithmetic is the stencil's. A
    gradient reads the stored Laplacians of every step once and writes them once."""
    size = 8 if c["dtype"] == "float64" else 4
    cells = (c["n0"] + 2 * c["layer"]) * (c["n1"] + 2 * c["layer"]) if c["absorbing"] != "none" else c["n0"] * c["n1"]
    sweep = cells * c["steps"] * c["shots"]
    trace = c["shots"] * c["recs"] * (c["steps"] // c["substeps"] + 1) * size
    flops = (2 * 2 * c["order"] + 6) * sweep
    if c["call"] == "forward":
        return {"bytes": c["n0"] * c["n1"] * size + trace, "flops": flops}
    history = 2 * sweep * size if c["storage"] == "autograd" else 0
    return {"bytes": 2 * c["n0"] * c["n1"] * size + 3 * trace + history,
            "flops": (2 if c["storage"] == "autograd" else 3) * flops + 2 * sweep}


def work(case):
    kind = case["kind"]
    if kind == "fwi":
        return _fwi_work(case)
    if kind == "batch":
        each = [_fwi_work(m) for m in _members(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if kind == "pat":
        # a volume does not fit on the chip: each step reads two levels and the medium and writes one
        cells = (case["n"] + 32) ** 3 * case["batch"] * case["steps"]
        sweeps = 2 if case["storage"] == "autograd" else 3
        return {"bytes": 16 * cells * sweeps, "flops": (2 * 3 * case["order"] + 6) * cells * sweeps}
    if kind == "reversal":
        cells = (case["n0"] + 20) * (case["n1"] + 20)
        return {"bytes": 4 * (case["n0"] * case["n1"] + case["recs"] * (case["steps"] + 1)), "flops": 22 * cells * case["steps"]}
    n = case["shots"] * case["recs"] * case["n_t"]
    length = 2 * case["n_t"]
    filters = 5  # the observation's low-pass; response, low-pass, low-pass, response of the residual
    size = 8 if case["dtype"] == "float64" else 4
    return {"bytes": 3 * n * size, "flops": int(filters * 2 * 2.5 * case["shots"] * case["recs"] * length * math.log2(length))}


# ------------------------------------------------------------------------------------------------
# the same passes in float64
# ------------------------------------------------------------------------------------------------
def _pad(x, a, mode):
    """The last ``len(a)`` axes of x extended by a[i] cells on both sides (zeros or the edge value)."""
    for k, w in enumerate(a):
        dim = x.ndim - len(a) + k
        n = x.shape[dim]
        idx = torch.arange(-w, n + w, device=x.device)
        y = x.index_select(dim, idx.clamp(0, n - 1))
        if mode == "zeros":
            keep = ((idx >= 0) & (idx < n)).to(x.dtype).view([-1 if d == dim else 1 for d in range(x.ndim)])
            y = y * keep
        x = y
    return x


def _depth(n, a, faces=False):
    pos = torch.arange(n + 2 * a + (1 if faces else 0), dtype=torch.float64, device=DEV) + (0.0 if faces else 0.5)
    return torch.clamp(torch.maximum(a - pos, pos - (a + n)), min=0.0) / max(a, 1)


def _shifted(p, dim, k):
    """p moved by k cells along dim, zeros entering."""
    n = p.shape[dim]
    z = torch.zeros_like(p.narrow(dim, 0, abs(k)))
    if k > 0:
        return torch.cat([p.narrow(dim, k, n - k), z], dim)
    return torch.cat([z, p.narrow(dim, 0, n + k)], dim)


def _laplacian(p, h, order):
    d = len(h)
    out = 0.0
    for ax in range(d):
        dim = p.ndim - d + ax
        one = _shifted(p, dim, 1) + _shifted(p, dim, -1)
        if order == 2:
            out = out + (one - 2.0 * p) / h[ax] ** 2
        else:
            two = _shifted(p, dim, 2) + _shifted(p, dim, -2)
            out = out + (-2.5 * p + (4.0 / 3.0) * one - two / 12.0) / h[ax] ** 2
    return out


def _points(pts, shape, a, h):
    """Flat indices and multilinear weights (n, 2^d) of points on the padded grid."""
    idx, wgt = torch.zeros(len(pts), 1, dtype=torch.long), torch.ones(len(pts), 1, dtype=torch.float64)
    P = [n + 2 * w for n, w in zip(shape, a)]
    for ax in range(len(shape)):
        u = ((pts[:, ax] + a[ax] * h[ax]) / h[ax] - 0.5).clamp(0.0, P[ax] - 1)
        i0 = torch.floor(u).clamp(max=P[ax] - 2).long()
        t = u - i0
        idx = (idx[:, :, None] * P[ax] + torch.stack([i0, i0 + 1], 1)[:, None, :]).flatten(1)
        wgt = (wgt[:, :, None] * torch.stack([1.0 - t, t], 1)[:, None, :]).flatten(1)
    return idx.to(DEV), wgt.to(DEV)


class _Scheme:
    """The leapfrog scheme on a padded grid in float64: a step function for autograd to differentiate."""

    def __init__(self, shape, a, h, order, absorbing, c_max, dt):
        self.shape, self.a, self.h, self.order, self.dt, self.kind = shape, a, h, order, dt, absorbing
        d, ln = len(shape), math.log(1e3)
        along = [[-1 if k == ax else 1 for k in range(d)] for ax in range(d)]
        self.pml = None
        if absorbing == "none":
            self.A = self.B = None
        elif absorbing == "cerjan":
            xi = [_depth(shape[k], a[k]).view(along[k]) for k in range(d)]
            self.A = self.B = torch.exp(-((0.3 * torch.maximum(xi[0] + 0 * xi[1], xi[1] + 0 * xi[0])) ** 2))
        elif absorbing == "sponge":
            s = sum(3.0 * c_max * ln / (a[k] * h[k]) * _depth(shape[k], a[k]).view(along[k]) ** 2 for k in range(d))
            self.A, self.B = 1.0 / (1.0 + 0.5 * dt * s), 1.0 - 0.5 * dt * s
        else:
            scale = [1.5 * c_max * ln / (a[k] * h[k]) for k in range(2)]
            zc = [scale[k] * _depth(shape[k], a[k]).view(along[k]) ** 2 for k in range(2)]
            zf = [scale[k] * _depth(shape[k], a[k], True).view(along[k]) ** 2 for k in range(2)]
            self.A, self.B = 1.0 / (1.0 + 0.5 * dt * (zc[0] + zc[1])), 1.0 - 0.5 * dt * (zc[0] + zc[1])
            self.zz = dt**2 * zc[0] * zc[1]
            den = [1.0 + 0.5 * dt * zf[k] for k in range(2)]
            self.pml = [((2.0 - den[k]) / den[k], dt * (zc[1 - k] - zf[k]) / (den[k] * h[k])) for k in range(2)]

    def padded(self):
        return [n + 2 * w for n, w in zip(self.shape, self.a)]

    def start(self, batch):
        P = self.padded()
        z = torch.zeros(batch, *P, device=DEV, dtype=torch.float64)
        if self.pml is None:
            return z, z
        return z, z, torch.zeros(batch, P[0] + 1, P[1], device=DEV, dtype=torch.float64), torch.zeros(
            batch, P[0], P[1] + 1, device=DEV, dtype=torch.float64)

    def step(self, state, C, n, source):
        prev, p = state[0], state[1]
        lap = _laplacian(p, self.h, self.order)
        faces = []
        if self.pml is not None:
            for ax in range(2):
                z = torch.zeros_like(p.narrow(1 + ax, 0, 1))
                alpha, beta = self.pml[ax]
                psi = alpha * state[2 + ax] + beta * torch.diff(torch.cat([z, p, z], 1 + ax), dim=1 + ax)
                lap = lap + 0.5 / self.h[ax] * torch.diff(psi + state[2 + ax], dim=1 + ax)
                faces.append(psi)
        B = 1.0 if self.B is None or (self.kind == "cerjan" and n == 0) else self.B
        new = 2.0 * p - B * prev + C * lap
        if self.pml is not None:
            new = new - self.zz * p
        if source is not None:
            idx, w = source
            new = new.flatten(1).scatter_add(1, idx, w(n)).view_as(new)
        return (p, new if self.A is None else self.A * new, *faces)


def _propagate(scheme, state, C, n_steps, sub, source, rec, cot, leaf):
    """Traces of a run and, with ``cot(traces)`` their cotangents, the gradient of the tensors ``leaf`` that
    C and the first state were made from: segments recomputed under autograd, last to first."""
    idx, wgt = rec

    def sample(p):
        return (p.flatten(1)[:, idx] * wgt).sum(-1)

    size = state[1].numel() * 8
    seg = max(2, min(40, int(1.5e9 / size)))
    made = state
    with torch.no_grad():
        Cd, st, keep, out = C.detach(), tuple(s.detach() for s in state), [], []
        for n in range(n_steps + 1):
            if n % seg == 0 and cot is not None:
                keep.append(st)
            if n % sub == 0:
                out.append(sample(st[1]))
            if n < n_steps:
                st = scheme.step(st, Cd, n, source)
        traces = torch.stack(out, -1)
    if cot is None:
        return traces, None
    g = cot(traces)
    gC, gst = torch.zeros_like(C), None
    for k in range(len(keep) - 1, -1, -1):
        with torch.enable_grad():
            first = tuple(s.detach().requires_grad_(True) for s in keep[k])
            Cl, st, total = C.detach().requires_grad_(True), None, 0.0
            st = first
            last = min((k + 1) * seg, n_steps + 1)
            for n in range(k * seg, last):
                if n % sub == 0:
                    total = total + (sample(st[1]) * g[..., n // sub]).sum()
                if n < n_steps:
                    st = scheme.step(st, Cl, n, source)
            if gst is not None:
                total = total + sum((s * v).sum() for s, v in zip(st, gst))
            if not torch.is_tensor(total):
                gst = tuple(torch.zeros_like(s) for s in first)
                continue
            got = torch.autograd.grad(total, (Cl, *first), allow_unused=True)
        gC = gC + (0 if got[0] is None else got[0])
        gst = tuple(torch.zeros_like(s) if v is None else v for s, v in zip(first, got[1:]))
    back = [(C, gC)] + list(zip(made, gst))
    back = [(t, v) for t, v in back if t.requires_grad]
    return traces, torch.autograd.grad([t for t, _ in back], leaf, [v for _, v in back])[0]


def _exact_fwi(case, prob):
    c, src, rec, n_t, obs = prob
    shape, h = (case["n0"], case["n1"]), (H, H)
    w = 0 if case["absorbing"] == "none" else case["layer"]
    a, sub = (w, w), case["substeps"]
    # the operator's own time step: the sampling interval over its stable substeps
    rho = 4.0 if case["order"] == 2 else 16.0 / 3.0
    stable = 0.9 * 2.0 / (C_MAX * math.sqrt(2 * rho / H**2))
    sub = max(1, math.ceil(_dt_obs(case) / stable - 1e-12))
    dt = _dt_obs(case) / sub
    scheme = _Scheme(shape, a, h, case["order"], case["absorbing"], C_MAX, dt)
    outs = []
    leaf = c.double().requires_grad_(case["call"] != "forward")
    C = _pad(leaf, a, "edge") ** 2 * dt**2
    si, sw = _points(src, shape, a, h)
    grad, traces = 0.0, []
    most = max(1, int(2.5e7 / (C.numel())))  # shots at a time
    for s0 in range(0, len(src), most):
        s1 = min(len(src), s0 + most)
        t0 = 1.2 / F0

        def wave(n, w=sw[s0:s1]):
            u = (math.pi * F0 * (n * dt - t0)) ** 2
            return w * ((1.0 - 2.0 * u) * math.exp(-u) * dt**2 / H**2)

        d = obs[s0:s1].double()
        tr, g = _propagate(scheme, scheme.start(s1 - s0), C, (n_t - 1) * sub, sub, (si[s0:s1], wave),
                           _points(rec, shape, a, h), None if case["call"] == "forward" else (lambda t, d=d: t - d), leaf)
        traces.append(tr)
        if g is not None:
            grad = grad + g
        if g is not None and s1 < len(src):
            C = _pad(leaf, a, "edge") ** 2 * dt**2
    outs = torch.cat(traces)
    return outs, grad, 0.5 * (outs - obs.double()).square().sum()


def _next_fast(n):
    while True:
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _filtered(x, length, window):
    f = torch.fft.rfftfreq(length, MISFIT_DT, device=DEV, dtype=torch.float64)
    return torch.fft.irfft(torch.fft.rfft(x, length) * window(f), length)[..., : x.shape[-1]]


def _lowpass(x):
    f1, f2 = (1 - MISFIT_TAPER) * MISFIT_FMAX, MISFIT_FMAX

    def window(f):
        roll = 0.5 * (1.0 + torch.cos(math.pi * (f - f1) / (f2 - f1)))
        return torch.where(f <= f1, torch.ones_like(f), torch.where(f < f2, roll, torch.zeros_like(f)))

    return _filtered(x, _next_fast(2 * x.shape[-1]), window)


def _exact_misfit(case, seed):
    pred, obs, mask = (t.double() for t in _misfit_inputs(case, seed))
    pred.requires_grad_(True)
    r = _filtered(pred, 2 * pred.shape[-1], lambda f: torch.exp(-0.5 * (f / MISFIT_SENSOR) ** 2)) - obs
    m = mask.expand_as(obs)
    loss = (m * _lowpass(r) ** 2).sum() / (m * _lowpass(obs) ** 2).sum()
    return {"loss": loss.detach(), "grad": torch.autograd.grad(loss, pred)[0]}


def _exact_pat(case, seed):
    c, p0, sensors, dt, obs = _pat_inputs(case, seed)
    n, a, h = case["n"], (16, 16, 16), (PAT_H,) * 3
    rho = 4.0 if case["order"] == 2 else 16.0 / 3.0
    c_max = float(c.max())
    sub = max(1, math.ceil(dt / (0.9 * 2.0 / (c_max * math.sqrt(3 * rho / PAT_H**2))) - 1e-12))
    dt = dt / sub
    scheme = _Scheme((n, n, n), a, h, case["order"], "sponge", c_max, dt)
    C = _pad(c, a, "edge") ** 2 * dt**2
    traces, grads = [], []
    for b in range(case["batch"]):
        leaf = p0[b:b + 1].double().requires_grad_(True)
        p = _pad(leaf, a, "zeros")
        d = obs[b:b + 1].double()
        tr, g = _propagate(scheme, (p + 0.5 * C * _laplacian(p, h, case["order"]), p), C, case["steps"] * sub, sub, None,
                           _points(sensors, (n, n, n), a, h), lambda t, d=d: t - d, leaf)
        traces.append(tr)
        grads.append(g)
    return {"traces": torch.cat(traces), "grad": torch.cat(grads)}


def _exact_reversal(case, seed):
    rec, dt, tr = _reversal_inputs(case, seed)
    shape, a, h, n_t = (case["n0"], case["n1"]), (10, 10), (PAT_H, PAT_H), case["steps"] + 1
    stable = 0.9 * 2.0 / (PAT_C * math.sqrt(2 * (16.0 / 3.0) / PAT_H**2))
    sub = max(1, math.ceil(dt / stable - 1e-12))
    scheme = _Scheme(shape, a, h, 4, "pml", PAT_C, dt / sub)
    C = torch.full(scheme.padded(), PAT_C**2 * (dt / sub) ** 2, device=DEV, dtype=torch.float64)
    cell = torch.floor((rec + torch.tensor(a) * PAT_H) / PAT_H).long()
    flat = (cell[:, 0] * scheme.padded()[1] + cell[:, 1]).tolist()
    last = {f: r for r, f in enumerate(flat)}
    where = torch.tensor(list(last), device=DEV)
    data = tr.double()[torch.tensor(list(last.values()), device=DEV)]

    def impose(p, n):
        u = (n_t - 1) - n / sub
        j = min(max(math.floor(u), 0), n_t - 1)
        k = min(j + 1, n_t - 1)
        p = p.clone()
        p.view(-1)[where] = (1.0 - (u - j)) * data[:, j] + (u - j) * data[:, k]
        return p

    st = scheme.start(1)
    st = (st[0], impose(st[1], 0), *st[2:])
    for n in range((n_t - 1) * sub):
        st = scheme.step(st, C, n, None)
        st = (st[0], impose(st[1], n + 1), *st[2:])
    return st[1][0, 10:10 + shape[0], 10:10 + shape[1]].clone()


def exact(case, seed):
    kind = case["kind"]
    if kind == "misfit":
        return _exact_misfit(case, seed)
    if kind == "pat":
        return _exact_pat(case, seed)
    if kind == "reversal":
        return _exact_reversal(case, seed)
    if kind == "batch":
        got = [_exact_fwi(m, _problem(m, seed, 100 * k)) for k, m in enumerate(_members(case, seed))]
        return {"loss": [x[2] for x in got], "grad": [x[1] for x in got]}
    traces, grad, loss = _exact_fwi(case, _problem(case, seed))
    if case["call"] == "forward":
        return traces
    return {"loss": loss, "grad": grad} if case["call"] == "graph" else {"traces": traces, "grad": grad}
