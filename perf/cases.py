"""Performance cases of the phase-field library: what a user's program has it do.

Each case is one pass through the public entry points (`Simulation`,
`Ensemble`, `adjoint.rollout`) on a state made from a seed:

  run       hand a microstructure over, advance it, take the fields back --
            one leg of a simulation between two outputs or checkpoints;
  ensemble  the same for a set of independent grain-growth runs of uneven
            sizes, advanced together;
  gradient  a differentiable rollout and its reverse sweep: the misfit of the
            final state against a target, differentiated with respect to the
            initial state and the three model parameters;
  analyse   the diagnostics of a snapshot: field sums and extremes, level
            set, grains, boundary lengths, per-tile ranges.

Sizes, coefficients, monitors and thresholds are those of the library's
presets, tuned configurations, benchmark and tests.  Runs are whole monitor
periods, so that a pass can be repeated from the same start.  Adaptive runs
hold FP32 and half data, and their fields are taken as float32; plain FP64
runs and the reference's own settings are taken as float64.
"""
import math

import numpy as np
import torch

import w3914777_gb300 as w
from w3914777_gb300 import adjoint, ensemble

MIX, PLAIN = w.END2END_MIX, w.PUREHIGH

# Tuned monitors: grain growth (single runs and ensembles) by the rate of
# change, Kobayashi and sintering by the spatial range; no FP64 above the
# FP32 tier where the tuner found none needed.
TUNED = {
    "graingrowth": {"monitor": w.MONITOR_RATE, "monitor_samples": 1, "monitor_field": -1, "thr_lo": 1e-5,
                    "thr_hi": 1e300, "tile": 32},
    "kobayashi": {"monitor": w.MONITOR_SPA, "monitor_samples": 1, "monitor_field": -1, "thr_lo": 0.05,
                  "thr_hi": 1e300, "tile": 32},
    "sintering": {"monitor": w.MONITOR_SPA, "monitor_samples": 1, "monitor_field": -1, "thr_lo": 1e-3,
                  "thr_hi": 0.9, "tile": 32},
}


def listed():
    return [
        # The headline: a 1024^2, eight-field coarsening run with the tuned monitor.
        {"name": "grains_1024_q8", "kind": "run", "model": "graingrowth", "preset": 0, "nx": 1024, "ny": 1024, "q": 8,
         "how": "tuned", "bc": 0, "steps": 500, "io": "f64", "out": "f32"},
        # The same run on a grid whose state is larger than the L2 cache.
        {"name": "grains_2048_q8", "kind": "run", "model": "graingrowth", "preset": 0, "nx": 2048, "ny": 2048, "q": 8,
         "how": "tuned", "bc": 0, "steps": 300, "io": "f64", "out": "f32"},
        # An odd-sided box with walls, six fields, the temporal monitor and a
        # float32 microstructure, as made in torch, to start from.
        {"name": "grains_odd_q6", "kind": "run", "model": "graingrowth", "preset": 0, "nx": 721, "ny": 397, "q": 6,
         "how": "temporal", "bc": 1, "steps": 300, "io": "f32", "out": "f32"},
        # The reference's own adaptive run: 512^2, two fields, 16^2 tiles,
        # half and FP64 tiles in the reference's order, 500 steps.
        {"name": "grains_reference_mix", "kind": "run", "model": "graingrowth", "preset": 1, "nx": 512, "ny": 512,
         "q": 2, "how": "reference", "bc": 0, "steps": 500, "io": "f64", "out": "f64"},
        # Plain FP64: what every adaptive result is judged against.
        {"name": "grains_fp64_q8", "kind": "run", "model": "graingrowth", "preset": 0, "nx": 512, "ny": 512, "q": 8,
         "how": "plain", "bc": 0, "steps": 100, "io": "f64", "out": "f64"},
        # The adaptive dendrite, zero flux, with the tuned monitor.
        {"name": "dendrite_512", "kind": "run", "model": "kobayashi", "preset": 0, "nx": 512, "ny": 512, "q": 2,
         "how": "tuned", "bc": 1, "steps": 500, "io": "f64", "out": "f32"},
        # The smallest run: a plain FP64 dendrite of a few tiles, where a step is latency.
        {"name": "dendrite_fp64_small", "kind": "run", "model": "kobayashi", "preset": 0, "nx": 128, "ny": 96, "q": 2,
         "how": "plain", "bc": 1, "steps": 200, "io": "f64", "out": "f64"},
        # Sintering of sixteen particles with the tuned monitor (FP64 interfaces, half bulk).
        {"name": "sintering_1024_n16", "kind": "run", "model": "sintering", "preset": 0, "nx": 1024, "ny": 1024,
         "q": 16, "how": "tuned", "bc": 0, "steps": 100, "io": "f64", "out": "f32"},
        # A parameter sweep: twelve uneven grain-growth runs advanced together.
        {"name": "ensemble_12", "kind": "ensemble", "members": 12, "lo": 128, "hi": 640, "steps": 200},
        # Gradients of a dendrite rollout, FP32, with the noise on (the differentiable-dendrite workload, fewer steps).
        {"name": "dendrite_gradient", "kind": "gradient", "model": "kobayashi", "nx": 256, "ny": 256, "q": 2, "bc": 1,
         "steps": 200, "dtype": "f32"},
        # Gradients of a grain-growth rollout in an odd-sided box with walls.
        {"name": "grains_gradient_odd", "kind": "gradient", "model": "graingrowth", "nx": 605, "ny": 443, "q": 8,
         "bc": 1, "steps": 40, "dtype": "f32"},
        # The diagnostics of a snapshot, as taken between two legs of a run.
        {"name": "microstructure_1024_q8", "kind": "analyse", "model": "graingrowth", "nx": 1024, "ny": 1024, "q": 8,
         "bc": 0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(rng, lo, hi, of=1):
    return max(of, int(round(_log(rng, lo, hi) / of)) * of)


def draw(rng):
    kind = rng.choice(["grains", "grains", "grains_plain", "grains_reference", "dendrite", "dendrite_plain", "sintering",
                       "sintering_plain", "ensemble", "dendrite_gradient", "grains_gradient", "analyse"])
    steps = 10 * int(round(_log(rng, 5, 40)))
    bc = rng.randrange(2)
    if kind == "grains":
        return {"kind": "run", "model": "graingrowth", "preset": 0, "nx": _side(rng, 128, 1400),
                "ny": _side(rng, 128, 1400), "q": rng.choice([2, 3, 4, 6, 8, 12, 16]),
                "how": rng.choice(["tuned", "tuned", "temporal"]), "bc": bc, "steps": steps,
                "io": rng.choice(["f32", "f64"]), "out": "f32"}
    if kind == "grains_plain":
        return {"kind": "run", "model": "graingrowth", "preset": 0, "nx": _side(rng, 64, 700),
                "ny": _side(rng, 64, 700), "q": rng.choice([2, 3, 4, 6, 8, 12]), "how": "plain", "bc": bc,
                "steps": steps, "io": "f64", "out": "f64"}
    if kind == "grains_reference":
        return {"kind": "run", "model": "graingrowth", "preset": rng.randint(1, 5), "nx": _side(rng, 128, 1024, 16),
                "ny": _side(rng, 128, 1024, 16), "q": 2, "how": "reference", "bc": 0, "steps": steps, "io": "f64",
                "out": "f64"}
    if kind == "dendrite":
        return {"kind": "run", "model": "kobayashi", "preset": 0, "nx": _side(rng, 96, 1400, 32),
                "ny": _side(rng, 96, 1400, 32), "q": 2, "how": "tuned", "bc": bc, "steps": steps,
                "io": rng.choice(["f32", "f64"]), "out": "f32"}
    if kind == "dendrite_plain":
        return {"kind": "run", "model": "kobayashi", "preset": rng.choice([0, 0, 2, 3, 4]),
                "nx": _side(rng, 64, 700, 32), "ny": _side(rng, 64, 700, 32), "q": 2, "how": "plain", "bc": bc,
                "steps": steps, "io": "f64", "out": "f64"}
    if kind == "sintering":
        return {"kind": "run", "model": "sintering", "preset": 0, "nx": _side(rng, 256, 1024, 32),
                "ny": _side(rng, 256, 1024, 32), "q": rng.randint(2, 16), "how": "tuned", "bc": bc,
                "steps": min(steps, 200), "io": "f64", "out": "f32"}
    if kind == "sintering_plain":
        return {"kind": "run", "model": "sintering", "preset": rng.choice([0, 1, 3]), "nx": _side(rng, 128, 640, 32),
                "ny": _side(rng, 128, 640, 32), "q": rng.choice([2, 2, 4, 7]), "how": "plain", "bc": bc,
                "steps": min(steps, 100), "io": "f64", "out": "f64"}
    if kind == "ensemble":
        return {"kind": "ensemble", "members": rng.randint(3, 24), "lo": 64, "hi": _side(rng, 160, 640),
                "steps": min(steps, 200)}
    if kind == "dendrite_gradient":
        return {"kind": "gradient", "model": "kobayashi", "nx": _side(rng, 48, 512), "ny": _side(rng, 48, 512), "q": 2,
                "bc": bc, "steps": min(steps, 200), "dtype": rng.choice(["f32", "f64"])}
    if kind == "grains_gradient":
        return {"kind": "gradient", "model": "graingrowth", "nx": rng.choice([_side(rng, 64, 640), _side(rng, 64, 640, 32)]),
                "ny": rng.choice([_side(rng, 64, 640), _side(rng, 64, 640, 32)]), "q": rng.choice([2, 4, 5, 8]), "bc": bc,
                "steps": rng.choice([16, 25, 40]), "dtype": rng.choice(["f32", "f64"])}
    return {"kind": "analyse", "model": "graingrowth", "nx": _side(rng, 200, 1600), "ny": _side(rng, 200, 1600),
            "q": rng.choice([2, 4, 6, 8, 12]), "bc": bc}


# ---- inputs -----------------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _grid(nx, ny, dev):
    y = torch.arange(ny, dtype=torch.float64, device=dev)[:, None]
    x = torch.arange(nx, dtype=torch.float64, device=dev)[None, :]
    return x, y


def _dist(x, y, cx, cy, nx, ny, bc):
    dx, dy = (x - cx).abs(), (y - cy).abs()
    if bc == 0:
        dx, dy = torch.minimum(dx, nx - dx), torch.minimum(dy, ny - dy)
    return torch.sqrt(dx * dx + dy * dy)


def _grains(nx, ny, q, bc, seed):
    """A polycrystal: a Voronoi tessellation whose cells each belong to one
    order parameter, with diffuse boundaries a few cells wide -- the state of
    a coarsening run past its first instants."""
    rng = np.random.default_rng(seed)
    dev = _dev()
    count = int(min(160, max(2 * q, nx * ny / 3600)))
    cx, cy = rng.uniform(0, nx, count), rng.uniform(0, ny, count)
    k = rng.permutation(np.arange(count) % q)
    x, y = _grid(nx, ny, dev)
    near = torch.full((q, ny, nx), 4.0 * (nx + ny), dtype=torch.float64, device=dev)
    for i in range(count):
        torch.minimum(near[k[i]], _dist(x, y, cx[i], cy[i], nx, ny, bc), out=near[k[i]])
    two = torch.topk(near, min(2, q), dim=0, largest=False).values
    if q == 1:
        return torch.ones_like(near)
    other = torch.where(near == two[0], two[1], two[0])  # the nearest site of any other field
    return 0.5 * (1 + torch.tanh((other - near) / 6.0))


def _dendrite(nx, ny, seed):
    """Solid nuclei with diffuse fronts in an undercooled melt that they have begun to heat."""
    rng = np.random.default_rng(seed)
    dev = _dev()
    x, y = _grid(nx, ny, dev)
    phi = torch.zeros(ny, nx, dtype=torch.float64, device=dev)
    heat = torch.zeros_like(phi)
    for _ in range(int(min(6, 1 + nx * ny // 40000))):
        cx, cy = rng.uniform(0.2, 0.8) * nx, rng.uniform(0.2, 0.8) * ny
        r = rng.uniform(5, 0.09 * min(nx, ny) + 5)
        d = torch.sqrt((x - cx) ** 2 + (1 + rng.uniform(0, 0.2)) * (y - cy) ** 2)
        phi = torch.maximum(phi, 0.5 * (1 - torch.tanh((d - r) / 1.7)))
        heat = torch.maximum(heat, rng.uniform(0.3, 0.6) * torch.exp(-((d - r) / 5.0) ** 2))
    return torch.stack([phi, heat])


def _particles(nx, ny, count, seed):
    """Discs that touch but do not overlap, each its own order parameter, with
    relaxed edges; the bulk of the particles and of the pores is exactly 1 and 0."""
    rng = np.random.default_rng(seed)
    dev = _dev()
    side = min(nx, ny)
    rs, cs = [], []
    rmax = min(40.0, 0.28 * side / math.sqrt(count))
    while len(rs) < count:
        r = rng.uniform(0.6 * rmax, rmax)
        for _ in range(400):
            if rs:
                j, th = rng.integers(len(rs)), rng.uniform(0, 2 * math.pi)
                c = (cs[j][0] + (r + rs[j]) * math.cos(th), cs[j][1] + (r + rs[j]) * math.sin(th))
            else:
                c = (0.5 * nx, 0.5 * ny)
            if not (r + 2 < c[0] < nx - r - 2 and r + 2 < c[1] < ny - r - 2):
                continue
            if all(math.hypot(c[0] - a[0], c[1] - a[1]) > r + b - 1e-6 for a, b in zip(cs, rs)):
                rs.append(r)
                cs.append(c)
                break
        else:
            rmax *= 0.9
    x, y = _grid(nx, ny, dev)
    f = torch.zeros(count + 1, ny, nx, dtype=torch.float64, device=dev)
    for i, (r, c) in enumerate(zip(rs, cs)):
        f[i + 1] = 0.5 * (1 - torch.tanh((torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2) - r) / 1.5))
    f[0] = f[1:].sum(0).clamp(max=1)
    f = torch.where(f < 1e-9, torch.zeros_like(f), torch.where(f > 1 - 1e-9, torch.ones_like(f), f))
    return f


def _initial(case, seed):
    if case["model"] == "graingrowth":
        return _grains(case["nx"], case["ny"], case["q"], case["bc"], seed)
    if case["model"] == "kobayashi":
        return _dendrite(case["nx"], case["ny"], seed)
    return _particles(case["nx"], case["ny"], case["q"], seed)


_DTYPE = {"f32": (torch.float32, w.F32), "f64": (torch.float64, w.F64)}


def _params(case):
    """Parameters of a run: a preset with this case's grid and monitor."""
    p = w.Params.preset(case["model"], case["preset"], nx=case["nx"], ny=case["ny"], bc=case["bc"], max_log=0)
    if case["model"] != "kobayashi":
        p.nfields = case["q"]
    p.noise = 0.0  # runs start from a given state; the gradient cases have the noise on
    if case["how"] == "plain":
        return p.replace(mode=PLAIN)
    if case["how"] == "reference":  # the reference's AMSTENCIL run with its Monitor2
        return p.replace(mode=MIX, monitor=w.MONITOR_TEM, thr_lo=1e-4, thr_hi=1e-4)
    if case["how"] == "temporal":  # three tiers by the change over a period, on the sample lattice
        return p.replace(mode=MIX, monitor=w.MONITOR_TEM, monitor_samples=0, monitor_field=-1, thr_lo=1e-4,
                         thr_hi=1e300, tile=32)
    return p.replace(mode=MIX, **TUNED[case["model"]])


def _member_params(case, seed):
    """An ensemble's members: uneven square grids, field counts and coefficients.
    The sizes and field counts are the case's, so that every seed has the same work."""
    shape = np.random.default_rng(1000 * case["members"] + case["hi"])
    rng = np.random.default_rng(seed)
    ps = []
    for _ in range(case["members"]):
        side = int(round(math.exp(shape.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        q = int(shape.choice([4, 8, 12, 16]))
        kappa, mobil = float(rng.uniform(1.0, 3.0)), float(rng.uniform(0.5, 2.0))
        p = w.Params.preset("graingrowth", 0, nx=side, ny=side, nfields=q, grcoef=kappa, mobil=mobil, mode=MIX,
                            max_log=0, **TUNED["graingrowth"])
        p.dt = ensemble.stable_dt(mobil, kappa, p.dx)
        ps.append(p)
    return ps


def _gradient_start(case, seed):
    """A rollout's start.  Kobayashi: the fronts on a slowly varying background,
    so that grad phi is nowhere lost in rounding: the anisotropy's angle, and
    with it the gradients, are well conditioned."""
    start = _initial(case, seed)
    if case["model"] == "kobayashi":
        x, y = _grid(case["nx"], case["ny"], start.device)
        start[0] = 0.02 + 0.94 * start[0] + 0.01 * torch.sin(0.11 * x) * torch.cos(0.09 * y)
    return start


def _gradient_params(case, seed):
    return w.Params.preset(case["model"], 0, nx=case["nx"], ny=case["ny"], bc=case["bc"], mode=PLAIN,
                           nfields=case["q"], seed=int(seed) + 1)


def _target(state, seed):
    """What a rollout is fitted to: the start, displaced by a few cells and dimmed."""
    rng = np.random.default_rng(seed + 77)
    return rng.uniform(0.8, 1.0) * torch.roll(state, (int(rng.integers(1, 5)), int(rng.integers(1, 5))), (-2, -1))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        dtype, code = _DTYPE[case["io"]]
        start = _initial(case, seed).to(dtype).contiguous()
        sim = w.Simulation(_params(case))
        out = torch.empty(start.shape, dtype=_DTYPE[case["out"]][0], device=start.device)
        torch.cuda.synchronize()
        return {"kind": kind, "sim": sim, "start": start, "code": code, "out": out, "out_code": _DTYPE[case["out"]][1],
                "steps": case["steps"]}
    if kind == "ensemble":
        ps = _member_params(case, seed)
        sims = [w.Simulation(p) for p in ps]
        starts = [_grains(p.nx, p.ny, p.nfields, 0, seed * 100 + i) for i, p in enumerate(ps)]
        outs = [torch.empty(s.shape, dtype=torch.float32, device=s.device) for s in starts]
        ens = w.Ensemble(sims)
        torch.cuda.synchronize()
        return {"kind": kind, "ens": ens, "sims": sims, "starts": starts, "outs": outs, "steps": case["steps"]}
    if kind == "gradient":
        p = _gradient_params(case, seed)
        dtype = _DTYPE[case["dtype"]][0]
        start = _gradient_start(case, seed)
        runner = adjoint.Rollout(p, case["steps"], dtype=dtype)
        values = torch.tensor([getattr(p, n) for n in adjoint.PARAM_NAMES[p.model]], dtype=dtype)
        state = {"kind": kind, "params": p, "steps": case["steps"], "runner": runner, "values": values,
                 "start": start.to(dtype).contiguous(), "target": _target(start, seed).to(dtype).contiguous()}
        torch.cuda.synchronize()
        return state
    p = w.Params.preset("graingrowth", 0, nx=case["nx"], ny=case["ny"], nfields=case["q"], bc=case["bc"], mode=PLAIN,
                        high_tier=w.TIER_FP32, max_log=0)
    sim = w.Simulation(p)
    start = _initial(case, seed)
    torch.cuda.synchronize()
    sim.set_fields_device(start.data_ptr(), w.F64)
    sim.synchronize()
    return {"kind": kind, "sim": sim, "q": case["q"]}


def run(state):
    kind = state["kind"]
    if kind == "run":
        sim = state["sim"]
        sim.set_fields_device(state["start"].data_ptr(), state["code"])
        sim.run(state["steps"])
        sim.get_fields_device(state["out"].data_ptr(), state["out_code"])
        return state["out"]
    if kind == "ensemble":
        for sim, start in zip(state["sims"], state["starts"]):
            sim.set_fields_device(start.data_ptr(), w.F64)
        state["ens"].run(state["steps"])
        state["ens"].synchronize()
        for sim, out in zip(state["sims"], state["outs"]):
            sim.get_fields_device(out.data_ptr(), w.F32)
        return state["outs"]
    if kind == "gradient":
        start = state["start"].detach().requires_grad_(True)
        values = state["values"].detach().clone().requires_grad_(True)
        final = adjoint.rollout(start, state["params"], state["steps"], param_values=values.double(),
                                runner=state["runner"])
        loss = 0.5 * (final - state["target"]).square().sum()
        loss.backward()
        return {"final": final.detach(), "grad_start": start.grad, "grad_values": values.grad}
    sim, q = state["sim"], state["q"]
    return {"sums": [sim.reduce(k, w.REDUCE_SUM) for k in range(q)],
            "extremes": [sim.reduce(0, w.REDUCE_MIN), sim.reduce(0, w.REDUCE_MAX)],
            "level_set": sim.interface(0, 0.5), "grains": sim.grains(0.5), "lengths": sim.boundary_lengths(),
            "ranges": sim.measure_tiles(w.MONITOR_SPA)}


# ---- the work that a pass cannot do without ----------------------------------

def work(case):
    """Bytes: each step reads the state once and writes it once, in the type
    that the run holds it in (adaptive runs: FP32 for grain growth, the half
    bulk of the dendrite and of sintering).  Operations: the update formula's."""
    kind = case["kind"]
    if kind == "ensemble":
        cf = sum(p.nx * p.ny * p.nfields for p in _member_params(case, 0))
        return {"bytes": cf * (case["steps"] * 8.0 + 12), "flops": cf * case["steps"] * 20.0}
    cells = case["nx"] * case["ny"]
    model, q = case["model"], case["q"]
    fields = 2 if model == "kobayashi" else q + 1 if model == "sintering" else q
    per = {"graingrowth": 20.0 * q, "kobayashi": 110.0, "sintering": 45.0 + 24.0 * q}[model]
    if kind == "analyse":
        return {"bytes": cells * q * 4.0, "flops": cells * q * 4.0}
    if kind == "gradient":
        size = 4 if case["dtype"] == "f32" else 8
        # forward, replay and adjoint step: 2, 2 and 3 passes over the state
        return {"bytes": cells * fields * size * 7.0 * case["steps"], "flops": cells * per * 4.0 * case["steps"]}
    held = 8 if case["how"] == "plain" else 4 if model == "graingrowth" and case["how"] != "reference" else 2
    moved = sum(4 if case[k] == "f32" else 8 for k in ("io", "out"))
    return {"bytes": cells * fields * (2.0 * held * case["steps"] + moved), "flops": cells * per * case["steps"]}


# ---- the same in 64 bits, in plain torch --------------------------------------

def _pad(f, r, bc):
    for d in (-1, -2):
        n = f.shape[d]
        a, b = f.narrow(d, 0, r), f.narrow(d, n - r, r)
        f = torch.cat([b, f, a] if bc == 0 else [a.flip(d), f, b.flip(d)], d)
    return f


class _Window:
    """Shifted views of a field padded by r cells."""

    def __init__(self, f, r, bc):
        self.f, self.r, self.ny, self.nx = _pad(f, r, bc), r, f.shape[-2], f.shape[-1]

    def __call__(self, kx, ky):
        return self.f[..., self.r + ky:self.r + ky + self.ny, self.r + kx:self.r + kx + self.nx]


def _grain_step(e, p, mobil, grcoef, gamma):
    s = _Window(e, 1, p.bc)
    lap = (s(-1, -1) + s(0, -1) + s(1, -1) + s(-1, 0) + s(1, 0) + s(-1, 1) + s(0, 1) + s(1, 1) - 8 * e) / (p.dx * p.dy)
    e2 = e * e
    dfd = e * (e2 - 1 + 2 * gamma * (e2.sum(0, keepdim=True) - e2))
    return e - p.dt * mobil * (dfd - grcoef * lap)


def _mix64(z):
    def lsr(v, k):
        return (v >> k) & ((1 << (64 - k)) - 1)
    z = z + (0x9E3779B97F4A7C15 - (1 << 64))
    z = (z ^ lsr(z, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    z = (z ^ lsr(z, 27)) * (0x94D049BB133111EB - (1 << 64))
    return z ^ lsr(z, 31)


def _noise(seed, step, shape, dev):
    """The driving term's noise: uniform in [0, 1) by step and cell (SplitMix64)."""
    one = torch.tensor([step], dtype=torch.int64, device=dev)
    key = _mix64(torch.tensor([seed], dtype=torch.int64, device=dev) ^ _mix64(one))
    z = _mix64(key + torch.arange(shape[0] * shape[1], dtype=torch.int64, device=dev))
    return (((z >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53).reshape(shape)


def _dendrite_step(state, p, delta, kappa, epsb, step):
    phi, T = state[0], state[1]
    sp, st = _Window(phi, 2, p.bc), _Window(T, 2, p.bc)
    px, py = (sp(1, 0) - sp(-1, 0)) * (0.5 / p.dx), (sp(0, 1) - sp(0, -1)) * (0.5 / p.dy)
    some = (px != 0) | (py != 0)  # no gradient: the angle counts as 0, and has no derivative
    a = p.aniso * (torch.atan2(torch.where(some, py, 0.0), torch.where(some, px, 1.0)) - p.theta0)
    eps = epsb * (1 + delta * torch.cos(a))
    epd = -epsb * p.aniso * delta * torch.sin(a)

    def lap(s, f):
        return (s(-1, 0) + s(1, 0) + s(-2, 0) + s(2, 0) + s(0, -1) + s(0, 1) + s(0, -2) + s(0, 2) - 8 * f) / (p.dx * p.dy)

    ty, tx = _Window(eps * epd * px, 1, p.bc), _Window(eps * epd * py, 1, p.bc)
    aniso = (ty(0, 1) - ty(0, -1)) * (0.5 / p.dy) - (tx(1, 0) - tx(-1, 0)) * (0.5 / p.dx)
    drive = phi - 0.5 + (p.alpha / p.pi) * torch.atan(p.gama * (p.teq - T))
    if p.noise != 0.0:
        drive = drive + p.noise * (_noise(p.seed, step, phi.shape, phi.device) - 0.5)
    d = (p.dt / p.tau) * (aniso + eps * eps * lap(sp, phi) + phi * (1 - phi) * drive)
    return torch.stack([phi + d, T + p.dt * lap(st, T) + kappa * d])


def _sintering_step(state, p):
    c, e = state[0], state[1:]
    s, inv = _Window(c, 1, p.bc), 1.0 / (p.dx * p.dy)
    s2, s3 = (e * e).sum(0), (e ** 3).sum(0)
    lap = (s(-1, 0) + s(1, 0) + s(0, -1) + s(0, 1) - 4 * c) * inv
    mu = p.B * (2 * c + 4 * s3 - 6 * s2) + 2 * p.A * c * (1 - c) * (1 - 2 * c) - 0.5 * p.coefm * lap
    m = _Window(mu, 1, p.bc)
    lapm = (m(-1, 0) + m(1, 0) + m(0, -1) + m(0, 1) - 4 * mu) * inv
    phi = c ** 3 * (10 - 15 * c + 6 * c * c)
    pairs = e.sum(0) ** 2 - s2 if e.shape[0] > 2 else 2 * e[0] * e[1] if e.shape[0] == 2 else torch.zeros_like(c)
    mob = p.dvol * phi + p.dvap * (1 - phi) + p.dsur * c * (1 - c) + p.dgrb * pairs
    cn = (c + p.dt * mob * lapm).clamp(0, 1)
    t = _Window(e, 1, p.bc)
    lape = (t(-1, 0) + t(1, 0) + t(0, -1) + t(0, 1) - 4 * e) * inv
    dfd = 12 * p.B * e * ((1 - cn) + s2 - e * (2 - cn))
    en = (e - p.dt * p.coefl * (dfd - 0.5 * p.coefk * lape)).clamp(0, 1)
    return torch.cat([cn[None], en])


def _advance(state, p, steps):
    for k in range(steps):
        if p.model == w.GRAINGROWTH:
            state = _grain_step(state, p, p.mobil, p.grcoef, p.gamma)
        elif p.model == w.KOBAYASHI:
            state = _dendrite_step(state, p, p.delta, p.kappa, p.epsb, k)
        else:
            state = _sintering_step(state, p)
    return state


def exact(case, seed):
    kind = case["kind"]
    if kind == "run":
        return _advance(_initial(case, seed).to(_DTYPE[case["io"]][0]).double(), _params(case), case["steps"])
    if kind == "ensemble":
        return [_advance(_grains(p.nx, p.ny, p.nfields, 0, seed * 100 + i), p, case["steps"])
                for i, p in enumerate(_member_params(case, seed))]
    if kind == "gradient":
        p, dtype = _gradient_params(case, seed), _DTYPE[case["dtype"]][0]
        start = _gradient_start(case, seed)
        target = _target(start, seed).to(dtype).double()
        start = start.to(dtype).double().requires_grad_(True)
        names = ("delta", "kappa", "epsb") if case["model"] == "kobayashi" else ("mobil", "grcoef", "gamma")
        v = [torch.tensor(getattr(p, n), dtype=dtype).double().to(start.device).requires_grad_(True) for n in names]
        state = start
        for k in range(case["steps"]):
            state = _dendrite_step(state, p, *v, k) if case["model"] == "kobayashi" else _grain_step(state, p, *v)
        (0.5 * (state - target).square().sum()).backward()
        return {"final": state.detach(), "grad_start": start.grad, "grad_values": torch.stack([x.grad for x in v])}
    f = _initial(case, seed).float().double()
    nx, ny, q, bc = case["nx"], case["ny"], case["q"], case["bc"]

    def edges(a, d):  # neighbouring pairs along one axis
        b = torch.roll(a, -1, d)
        return (a, b) if bc == 0 else (a.narrow(d, 0, a.shape[d] - 1), b.narrow(d, 0, a.shape[d] - 1))

    solid = f[0] >= 0.5
    level = {"cells": None, "area": float(solid.sum()), "xmin": None, "xmax": None, "ymin": None, "ymax": None,
             "perimeter": float(sum((a != b).sum() for a, b in (edges(solid, 0), edges(solid, 1))))}
    lab = f.argmax(0)
    pair = torch.zeros(q * q, dtype=torch.float64, device=f.device)
    for a, b in (edges(lab, 0), edges(lab, 1)):
        m = a != b
        pair += torch.bincount((torch.minimum(a, b) * q + torch.maximum(a, b))[m], minlength=q * q).double()
    pair = pair.reshape(q, q)
    T = 32
    g = f
    hi = torch.nn.functional.max_pool2d(g, T, ceil_mode=True)
    lo = -torch.nn.functional.max_pool2d(-g, T, ceil_mode=True)
    return {"sums": f.sum((1, 2)).tolist(), "extremes": [float(f[0].min()), float(f[0].max())], "level_set": level,
            "grains": {"grains": None, "cells": None, "mean_area": None}, "lengths": (pair + pair.T).cpu().numpy(),
            "ranges": (hi - lo).amax(0).cpu().numpy()}
