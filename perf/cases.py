"""The workloads whose speed counts, each through the public entry points of physica_b200.

The states are fluid in motion rather than the lattice at rest: a block of fluid at the dam-break
spacing (half the support radius), every particle moved off its lattice point by up to `jitter`
support radii, a sheared velocity field with Gaussian noise, and for the PBF forward steps a thin
spray of single particles above the block.  Parameters are the ones of the dam-break scenes
(physica_b200/scenes.py).  Everything is drawn on the GPU from the seed.

Kinds:
  step     one PBF substep (PBF.forward_step)
  host     one PBF substep over host arrays (PBF.forward_step_host)
  batch    one substep of many scenes of mixed sizes (Batch.forward_step)
  grad     one gradient step: differentiable substep and its adjoint (forward_step, vjp_step)
  tangent  one tangent step: differentiable substep and its tangent (forward_step, jvp_step)
  rollout  loss and gradients of a checkpointed rollout of a batch (trajectory.loss_and_gradients)
  sph      one SPH substep (SPH.forward_step)
  sph_grad one SPH gradient step (forward_step, vjp_step)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from physica_b200 import pbf, sph, trajectory

F32 = np.float32
PI = float(F32(3.14159265358979323846))
METHODS = ("wcsph", "pcisph", "iisph", "dfsph")


# ----------------------------------------------------------------------------------- the cases
def _case(name, kind, nx, ny, nz, *, h=0.025, iterations=4, launch="default", scenes=1, low=0, jitter=0.15, dt=1.0 / 120.0,
          post=True, scorr=False, boundary=False, method="", steps=1, every=1):
    return {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "h": h, "iterations": iterations, "launch": launch,
            "scenes": scenes, "low": low, "jitter": jitter, "dt": dt, "post": post, "scorr": scorr, "boundary": boundary,
            "method": method, "steps": steps, "every": every}


def listed():
    return [
        # the dam-break example (python -m physica_b200.simulation): one step of 5,376 particles
        # with the solver as it is constructed; launches and latency count
        _case("example_step_5k", "step", 16, 28, 12, h=0.05, iterations=5, jitter=0.05, dt=1.0 / 240.0, post=False),
        # an interactive scene: 32,768 particles stepped by graph replay
        _case("step_32k", "step", 32, 32, 32, launch="graph"),
        # the large dam break: 1,048,576 particles, eight iterations, autotuned and graph-replayed
        _case("step_1m", "step", 128, 64, 128, iterations=8, launch="tuned"),
        # an odd-sized scene between two plates of boundary particles, with artificial pressure
        _case("boundary_step_103k", "step", 47, 53, 41, scorr=True, boundary=True),
        # a host program without device buffers: upload, step, download
        _case("host_step_262k", "host", 64, 64, 64, launch="graph"),
        # many scenes at once (dataset generation): 64 scenes of 2,048 to 65,536 particles
        _case("batch_step_64", "batch", 0, 0, 0, scenes=64, low=2048, launch="tuned"),
        # training through one substep: 65,536 particles, every parameter's adjoint
        _case("grad_step_64k", "grad", 32, 64, 32),
        # trajectory optimisation of several scenes: checkpointed rollouts with recomputation.  Few
        # steps of an inviscid scene near the lattice: the gradient of a longer or rougher rollout
        # changes by more than itself when the inputs' last bits do
        _case("batch_rollout_8", "rollout", 0, 0, 0, scenes=8, low=16384, jitter=0.05, post=False, steps=4, every=2),
        # forward-mode sensitivity of the large scene
        _case("tangent_step_1m", "tangent", 128, 64, 128),
        # weakly compressible SPH at one million particles
        _case("wcsph_step_1m", "sph", 128, 64, 128, jitter=0.05, dt=4e-4, method="wcsph"),
        # the divergence-free solver on an odd-sized block, warm-started
        _case("dfsph_step_270k", "sph", 75, 60, 60, jitter=0.05, dt=4e-4, method="dfsph"),
        # training through a pressure solve
        _case("pcisph_grad_131k", "sph_grad", 64, 32, 64, jitter=0.05, dt=4e-4, method="pcisph"),
    ]


# particle counts that a drawn case of a kind spans
_RANGE = {"step": (512, 1 << 20), "host": (4096, 1 << 20), "batch": (8, 64), "grad": (2048, 1 << 18), "tangent": (2048, 1 << 19),
          "rollout": (2, 8), "sph": (4096, 1 << 20), "sph_grad": (2048, 1 << 17)}


def draw(rng):
    kind = rng.choice(("step", "step", "step", "host", "batch", "grad", "tangent", "rollout", "sph", "sph", "sph_grad"))
    lo, hi = _RANGE[kind]
    size = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind in ("batch", "rollout"):
        return _drawn(kind, 0, 0, 0, scenes=size, low=rng.choice((2048, 4096, 16384)) if kind == "batch" else 16384,
                      launch=rng.choice(("default", "graph", "tuned")) if kind == "batch" else "default",
                      iterations=rng.randint(2, 4), steps=rng.randint(2, 4), every=rng.randint(1, 3), post=kind == "batch",
                      jitter=0.15 if kind == "batch" else 0.05)
    # a block of about `size` particles with uneven, often odd, sides
    nx = max(4, int(round(size ** (1.0 / 3.0) * rng.uniform(0.7, 1.4))))
    ny = max(4, int(round(math.sqrt(size / nx) * rng.uniform(0.8, 1.25))))
    nz = max(4, size // (nx * ny))
    if kind in ("sph", "sph_grad"):
        return _drawn(kind, nx, ny, nz, jitter=0.05, dt=4e-4, method=rng.choice(METHODS))
    return _drawn(kind, nx, ny, nz, h=rng.choice((0.025, 0.05, 0.1)), iterations=rng.randint(1, 6 if kind in ("step", "host") else 4), jitter=rng.choice((0.05, 0.15)),
                  launch=rng.choice(("default", "graph", "tuned")) if kind in ("step", "host") else "default",
                  post=rng.random() < 0.8, scorr=rng.random() < 0.3, boundary=kind in ("step", "grad") and rng.random() < 0.2)


def _drawn(kind, nx, ny, nz, **options):
    case = _case("", kind, nx, ny, nz, **options)
    del case["name"]
    return case


# ------------------------------------------------------------------------------------- inputs
def _counts(case, seed):
    """Scene sizes of a batch: log-uniform from `low` to 32 (8 for a rollout) times as many."""
    span = 8 if case["kind"] == "rollout" else 32
    # the sizes stand for the batch's make-up, not for its data: spread evenly over the logarithm
    k = case["scenes"]
    return [int(round(case["low"] * span ** ((s * 7 % k + 0.5) / k))) | 1 for s in range(k)]


def _block(nx, ny, nz, h, dt, spray, case, generator, count=None):
    """Positions and velocities (3, N) of one block of moving fluid, its box, and the time step."""
    dev = "cuda"
    spacing = 0.5 * h
    k, j, i = torch.meshgrid(torch.arange(nz, device=dev), torch.arange(ny, device=dev), torch.arange(nx, device=dev), indexing="ij")
    x = torch.stack([i.reshape(-1), j.reshape(-1), k.reshape(-1)]).double()
    if count is not None:
        x = x[:, :count]
    n = x.shape[1]
    u = torch.rand((3, n), generator=generator, device=dev, dtype=torch.float64)
    x = (x + 1.0) * spacing + (2.0 * u - 1.0) * (case["jitter"] * h)
    hi = [2.0 * (nx + 2) * spacing, 2.0 * (ny + 2) * spacing, 1.5 * (nz + 2) * spacing]
    sides = torch.tensor(hi, device=dev, dtype=torch.float64)[:, None]
    if spray:   # one particle in two hundred flies alone above the block
        fly = torch.arange(0, n, 200, device=dev)
        u = torch.rand((3, fly.numel()), generator=generator, device=dev, dtype=torch.float64)
        u[1] = 0.55 + 0.4 * u[1]
        x[:, fly] = u * sides
    noise = torch.randn((3, n), generator=generator, device=dev, dtype=torch.float64)
    v = 0.1 * noise
    v[0] += 0.5 * x[1] / sides[1]
    v[1] -= 0.3 * x[0] / sides[0]
    return x.float().contiguous(), v.float().contiguous(), hi


def _plates(h, hi, x):
    """A sliding floor under the block and a static wall beside it (lattices at half the support radius)."""
    s = 0.5 * h
    top = [float(x[a].max()) for a in range(3)]
    right = float(x[0].median()) * 2.0
    out = []
    for a in np.arange(s, min(hi[0], 2.0 * right), s):
        for c in np.arange(s, min(hi[2], top[2] + s), s):
            out.append(((float(F32(a)), float(F32(0.3 * s)), float(F32(c))), (float(F32(0.05)), 0.0, 0.0), float(F32(s ** 3))))
    for b in np.arange(s, 0.5 * hi[1], s):
        for c in np.arange(s, min(hi[2], top[2] + s), s):
            out.append(((float(F32(right + 2.0 * s)), float(F32(b)), float(F32(c))), (0.0, 0.0, 0.0), float(F32(s ** 3))))
    return out


def _inputs(case, seed):
    """What both the framework and the 64-bit restatement start from."""
    generator = torch.Generator(device="cuda")
    generator.manual_seed(1000003 * seed + 17)
    h, dt = float(F32(case["h"])), float(F32(case["dt"]))
    is_sph = case["kind"] in ("sph", "sph_grad")
    scenes = []
    if case["kind"] in ("batch", "rollout"):
        for count in _counts(case, seed):
            nx = max(2, math.ceil((count / 2.0) ** (1.0 / 3.0)))
            ny = math.ceil(count / (nx * nx))
            scenes.append(_block(nx, ny, nx, h, dt, case["kind"] == "batch", case, generator, count))
    else:
        scenes.append(_block(case["nx"], case["ny"], case["nz"], h, dt, case["kind"] in ("step", "host"), case, generator))
    x = torch.cat([s[0] for s in scenes], 1).contiguous()
    v = torch.cat([s[1] for s in scenes], 1).contiguous()
    n = x.shape[1]
    volume = F32(0.5 * h) ** 3
    full = lambda value: torch.full((n,), float(F32(value)), dtype=torch.float32, device="cuda")
    if is_sph:
        wc = case["method"] == "wcsph"
        parameters = {"masses": full(1000.0 * volume), "rest_densities": full(1000.0), "viscosities": full(0.05 if wc else 0.001),
                      "surface_tensions": full(0.05), "speed_of_sound": full(20.0), "tait_exponent": full(7.0),
                      "boundary_surface_tension": full(0.02), "pressure_relaxation": full(0.5), "jacobi_relaxation": full(0.5),
                      "divergence_relaxation": full(0.5), "density_relaxation": full(0.5)}
    else:
        post = 1.0 if case["post"] else 0.0
        parameters = {"masses": full(1000.0 * volume), "rest_densities": full(1000.0), "relaxation": full(1000.0),
                      "artificial_pressure_strength": full(1e-5 if case["scorr"] else 0.0), "artificial_pressure_exponent": full(4.0),
                      "artificial_pressure_radius": full(0.3 * h), "xsph_viscosity": full(post * 0.01 * volume),
                      "vorticity_confinement": full(post * 1e-4 * volume)}
    noise = lambda *shape: torch.randn(shape, generator=generator, device="cuda", dtype=torch.float64)
    control = (0.05 * noise(3, n)).float()
    out = {"x": x, "v": v, "control": control, "parameters": parameters, "boxes": [s[2] for s in scenes],
           "counts": [s[0].shape[1] for s in scenes], "h": h, "dt": dt, "plates": []}
    if case["boundary"]:
        out["plates"] = _plates(h, out["boxes"][0], x)
    if case["kind"] in ("grad", "sph_grad"):   # the adjoint of a loss over the next state
        out["adjoint"] = (noise(3, n), 1e-2 * noise(3, n))
    if case["kind"] == "tangent":              # a direction in initial state and controls
        out["tangent"] = (h * noise(3, n).float(), noise(3, n).float(), noise(3, n).float())
    if case["kind"] == "rollout":
        out["targets"] = (x + h * noise(3, n).float()).contiguous()
    if case["method"] == "dfsph":
        rnd = lambda: 50.0 * torch.rand(n, generator=generator, device="cuda", dtype=torch.float64).float()
        out["warm"] = (rnd(), rnd())
    return out


def _domain(case, data, scene):
    h = data["h"]
    box = pbf.BoxBoundary((0.0, 0.0, 0.0), tuple(float(F32(b)) for b in data["boxes"][scene]))
    return pbf.DomainConfiguration(data["counts"][scene], data["dt"], h, float(F32(0.2) * F32(h)), (0.0, float(F32(-9.8)), 0.0), box,
                                   data["plates"])


def prepare(case, seed):
    data = _inputs(case, seed)
    kind = case["kind"]
    differentiable = kind in ("grad", "tangent", "rollout", "sph_grad")
    mode = pbf.ExecutionMode.differentiable if differentiable else pbf.ExecutionMode.forward
    s = {"kind": kind, "case": case}
    control = pbf.Control(data["control"])
    if kind in ("sph", "sph_grad"):
        solver = sph.SPH(_domain(case, data, 0), sph.Configuration(method=sph.Method[case["method"]]), mode)
        state = solver.allocate_state()
        state.positions.copy_(data["x"])
        state.velocities.copy_(data["v"])
        if "warm" in data:
            state.warm_divergence_pressure.copy_(data["warm"][0])
            state.warm_density_pressure.copy_(data["warm"][1])
        parameters = sph.Parameters(data["parameters"])
        s.update(next=solver.allocate_state(), cache=solver.allocate_step_cache())
    elif kind in ("batch", "rollout"):
        solver = pbf.Batch([_domain(case, data, k) for k in range(len(data["counts"]))], pbf.Configuration(case["iterations"], 2), mode)
        state = pbf.State(data["x"], data["v"], 0)
        parameters = pbf.Parameters(data["parameters"])
        if kind == "batch":
            solver.reserve_caches(1)
            s["next"] = solver.allocate_state()
        else:
            s["targets"] = data["targets"]
            s["rollout"] = trajectory.Rollout(solver, control, parameters, case["steps"], min(case["every"], case["steps"]))
    else:
        solver = pbf.PBF(_domain(case, data, 0), pbf.Configuration(case["iterations"], 2), mode)
        state = pbf.State(data["x"], data["v"], 0)
        parameters = pbf.Parameters(data["parameters"])
        s.update(next=solver.allocate_state(), cache=solver.allocate_step_cache())
    s.update(solver=solver, state=state, control=control, parameters=parameters)
    if case["launch"] == "tuned":
        solver.autotune(state, control, parameters, repeats=2)
    if kind in ("step", "host", "batch") and case["launch"] != "default":
        solver.set_graph_mode(True)
    if kind == "host":
        pin = lambda t: t.cpu().pin_memory()
        s["host"] = [pin(data["x"]), pin(data["v"]), pin(torch.zeros_like(data["x"])), pin(torch.zeros_like(data["v"]))]
    if kind in ("grad", "sph_grad"):
        if kind == "grad":
            s["next_adjoint"] = pbf.StateAdjoint(*data["adjoint"])
        else:
            s["next_adjoint"] = sph.StateAdjoint(*data["adjoint"])
            if case["method"] == "dfsph":
                zero = lambda: torch.zeros(solver.count, dtype=torch.float64, device="cuda")
                s["next_adjoint"] = sph.StateAdjoint(*data["adjoint"], zero(), zero())
        s.update(previous=solver.allocate_state_adjoint(), control_adjoint=solver.allocate_control_adjoint(),
                 parameter_adjoint=solver.allocate_parameter_adjoint())
    if kind == "tangent":
        dx, dv, da = data["tangent"]
        s.update(state_tangent=pbf.StateTangent(dx, dv), control_tangent=pbf.Control(da),
                 parameter_tangent=solver.allocate_parameter_tangent(), next_tangent=solver.allocate_state_tangent())
    return s


# ------------------------------------------------------------------------------------ one pass
_PBF_ADJOINTS = ("masses", "rest_densities", "relaxation", "artificial_pressure_strength", "xsph_viscosity", "vorticity_confinement")
_SPH_ADJOINTS = {"wcsph": ("masses", "rest_densities", "viscosities", "surface_tensions", "speed_of_sound", "tait_exponent"),
                 "pcisph": ("masses", "rest_densities", "viscosities", "pressure_relaxation"),
                 "iisph": ("masses", "rest_densities", "viscosities", "jacobi_relaxation"),
                 "dfsph": ("masses", "rest_densities", "viscosities", "divergence_relaxation", "density_relaxation")}


def run(s):
    kind, solver = s["kind"], s["solver"]
    state, control, parameters = s["state"], s["control"], s["parameters"]
    if kind == "host":
        x, v, xo, vo = s["host"]
        solver.forward_step_host(x, v, control, parameters, xo, vo, s["cache"], 0)
        return {"positions": xo, "velocities": vo}
    if kind == "rollout":
        g = trajectory.loss_and_gradients(solver, state, control, parameters, s["targets"], s["rollout"].steps, s["rollout"].every,
                                          s["rollout"])
        return {"losses": torch.tensor(g.loss, dtype=torch.float64), "positions": s["rollout"].final.positions,
                "initial_positions": g.initial_positions, "initial_velocities": g.initial_velocities, "controls": g.controls}
    following = s["next"]
    solver.forward_step(state, control, parameters, following, 0 if kind == "batch" else s["cache"])
    out = {"positions": following.positions, "velocities": following.velocities}
    if kind == "sph" and s["case"]["method"] == "dfsph":
        out["divergence_pressure"] = following.warm_divergence_pressure
        out["density_pressure"] = following.warm_density_pressure
    if kind in ("grad", "sph_grad"):
        previous, ca, pa = s["previous"], s["control_adjoint"], s["parameter_adjoint"]
        previous.positions.zero_()
        previous.velocities.zero_()
        ca.external_accelerations.zero_()
        names = _PBF_ADJOINTS if kind == "grad" else _SPH_ADJOINTS[s["case"]["method"]]
        for name in names:
            pa.tensors[name].zero_()
        solver.vjp_step(state, control, parameters, following, s["cache"], s["next_adjoint"], previous, ca, pa)
        out.update(position_adjoint=previous.positions, velocity_adjoint=previous.velocities, control_adjoint=ca.external_accelerations)
        out.update({name + "_adjoint": pa.tensors[name] for name in names})
    if kind == "tangent":
        t = s["next_tangent"]
        solver.jvp_step(state, control, parameters, following, s["cache"], s["state_tangent"], s["control_tangent"],
                        s["parameter_tangent"], t)
        out.update(position_tangent=t.positions, velocity_tangent=t.velocities)
    return out


def _particles(case):
    if case["kind"] in ("batch", "rollout"):
        return sum(_counts(case, 0))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    n, k, kind = _particles(case), case["iterations"], case["kind"]
    pairs = 33.0 * n   # neighbours within the support at the block's spacing
    if kind in ("sph", "sph_grad"):
        passes = {"wcsph": 3.0, "pcisph": 2.0 + 12.0, "iisph": 2.0 + 12.0, "dfsph": 4.0 + 20.0}[case["method"]]
        forward = 25.0 * passes * pairs
        state = 24.0 if case["method"] != "dfsph" else 32.0
        data = n * (2.0 * state + 12.0 + 4.0 * len(_SPH_ADJOINTS[case["method"]]))
    else:
        forward = (69.0 * k + 81.0) * pairs
        data = n * (48.0 + 12.0 + 32.0)
    if kind in ("step", "host", "batch", "sph"):
        return {"bytes": data, "flops": forward}
    if kind == "tangent":
        return {"bytes": data + n * 60.0, "flops": 3.0 * forward}
    adjoints = len(_PBF_ADJOINTS) if kind != "sph_grad" else len(_SPH_ADJOINTS[case["method"]])
    if kind in ("grad", "sph_grad"):
        return {"bytes": data + n * (48.0 + 2.0 * (72.0 + 8.0 * adjoints)), "flops": 4.0 * forward}
    # every step's forward and adjoint; checkpoints and recomputation are the method's own
    return {"bytes": case["steps"] * n * 24.0 + n * (32.0 + 12.0 + 72.0), "flops": case["steps"] * 4.0 * forward}


def tolerance(case):
    """About four times the largest error against exact() that was seen over the range (32-bit
    arithmetic throughout; velocities divide a position change by the time step, and adjoints and
    tangents by pair distances).  A rollout's is four times the change that a flip of its inputs'
    last bits makes, 1.4e-2 for four steps."""
    kind = case["kind"]
    if kind in ("step", "host", "batch"):
        return {"rel": 1.5e-4 if case["iterations"] <= 6 else 4e-4}
    if kind == "sph":
        return {"rel": 1e-5 if case["method"] == "wcsph" else 6e-4}
    return {"rel": {"grad": 2.4e-3, "sph_grad": 2.4e-3, "tangent": 1.2e-2, "rollout": 5e-2}[kind]}


# ----------------------------------------------------------------- the same, in 64 bits and torch
class _Pairs:
    """Candidate pairs of the 27-cell stencil of the positions `at` (home cells are fixed for the
    step); `within(x)` gives the pairs (i, j) of it that are inside the support at positions x."""

    def __init__(self, at, others, h, box):
        dims = [int(np.ceil(F32(F32(b) - F32(0.0)) / F32(h))) for b in box]
        self.h, self.dims = h, dims
        cell = lambda p: [torch.clamp(torch.floor(p[a].float() / torch.tensor(h, device=p.device, dtype=torch.float32)), 0, dims[a] - 1).long()
                          for a in range(3)]
        self.home = cell(at)
        key = cell(others)
        flat = (key[0] * dims[1] + key[1]) * dims[2] + key[2]
        self.order = torch.argsort(flat, stable=True)
        counts = torch.bincount(flat, minlength=dims[0] * dims[1] * dims[2])
        self.start = torch.cat([torch.zeros(1, dtype=torch.long, device=at.device), torch.cumsum(counts, 0)])

    @torch.no_grad()
    def within(self, x, y):
        n = x.shape[1]
        found_i, found_j = [], []
        for first in range(0, n, 1 << 17):
            rows = torch.arange(first, min(n, first + (1 << 17)), device=x.device)
            for ox in (-1, 0, 1):
                for oy in (-1, 0, 1):
                    cx, cy = self.home[0][rows] + ox, self.home[1][rows] + oy
                    ok = (cx >= 0) & (cy >= 0) & (cx < self.dims[0]) & (cy < self.dims[1])
                    cx, cy = cx.clamp(0, self.dims[0] - 1), cy.clamp(0, self.dims[1] - 1)
                    z0 = (self.home[2][rows] - 1).clamp(min=0)
                    z1 = (self.home[2][rows] + 1).clamp(max=self.dims[2] - 1)
                    base = (cx * self.dims[1] + cy) * self.dims[2]
                    b = self.start[base + z0]
                    length = torch.where(ok, self.start[base + z1 + 1] - b, torch.zeros_like(b))
                    total = torch.cumsum(length, 0)
                    i = torch.repeat_interleave(rows, length)
                    slot = torch.arange(i.numel(), device=x.device) - torch.repeat_interleave(total - length, length) \
                        + torch.repeat_interleave(b, length)
                    j = self.order[slot]
                    d = x[:, i] - y[:, j]
                    keep = (d * d).sum(0) < self.h * self.h
                    found_i.append(i[keep])
                    found_j.append(j[keep])
        return torch.cat(found_i), torch.cat(found_j)


def _sum(i, values, n):
    if values.dim() == 1:
        return torch.zeros(n, dtype=values.dtype, device=values.device).index_add(0, i, values)
    return torch.stack([_sum(i, values[a], n) for a in range(values.shape[0])])


def _safe_norm(d):
    r2 = (d * d).sum(0)
    zero = r2 == 0
    return torch.where(zero, torch.zeros_like(r2), torch.sqrt(torch.where(zero, torch.ones_like(r2), r2)))


def _poly6(r2, h):
    return 315.0 * (h * h - r2).clamp(min=0.0) ** 3 / (64.0 * PI * h ** 9)


def _spiky(d, h):
    r = _safe_norm(d)
    zero = r == 0
    s = -45.0 / (PI * h ** 6) * (h - r) ** 2 / torch.where(zero, torch.ones_like(r), r)
    return d * torch.where(zero, torch.zeros_like(s), s)


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _clamped(x, box, radius):
    lo = float(F32(0.0) + F32(radius))
    return torch.stack([x[a].clamp(lo, float(F32(box[a]) - F32(radius))) for a in range(3)])


def _pbf_substep(x, v, control, p, h, dt, box, radius, iterations, plates):
    n = x.shape[1]
    gravity = torch.tensor([0.0, float(F32(-9.8)), 0.0], dtype=x.dtype, device=x.device)[:, None]
    star = x + dt * v + dt * dt * (gravity + control)
    with torch.no_grad():
        at = star.detach()
        grid = _Pairs(at, at, h, box)
        if plates:
            t = float(F32(1) * F32(dt))
            bx = torch.tensor([[q[0][a] + t * q[1][a] for q in plates] for a in range(3)], dtype=x.dtype, device=x.device)
            bvol = torch.tensor([q[2] for q in plates], dtype=x.dtype, device=x.device)
            bgrid = _Pairs(at, bx, h, box)
    detached = lambda t: torch.autograd.forward_ad.unpack_dual(t).primal.detach()
    mass, rest = p["masses"], p["rest_densities"]
    y = star
    for _ in range(iterations):
        i, j = grid.within(detached(y), detached(y))
        other = i != j
        density = _sum(i, mass[j] * _poly6(((y[:, i] - y[:, j]) ** 2).sum(0), h), n)
        i, j = i[other], j[other]
        d = y[:, i] - y[:, j]
        g = _spiky(d, h)
        c = mass[j] / rest[i]
        total = _sum(i, c * g, n)
        denominator = p["relaxation"] + _sum(i, c * c * (g * g).sum(0), n)
        if plates:
            bi, bj = bgrid.within(detached(y), bx)
            bd = y[:, bi] - bx[:, bj]
            bg = _spiky(bd, h)
            density = density + _sum(bi, rest[bi] * bvol[bj] * _poly6((bd * bd).sum(0), h), n)
            total = total + _sum(bi, bvol[bj] * bg, n)
        denominator = denominator + (total * total).sum(0)
        lam = -(density / rest - 1.0) / denominator

        def scorr(i, r2):
            w = _poly6(r2, h)
            ratio = w / _poly6(p["artificial_pressure_radius"] ** 2, h)[i]
            return -p["artificial_pressure_strength"][i] * ratio ** p["artificial_pressure_exponent"][i]

        factor = c * (lam[i] + lam[j] + scorr(i, (d * d).sum(0)))
        step = _sum(i, factor * g, n)
        if plates:
            step = step + _sum(bi, bvol[bj] * (lam[bi] + scorr(bi, (bd * bd).sum(0))) * bg, n)
        y = _clamped(y + step, box, radius)
    velocity = (y - x) / dt
    i, j = grid.within(detached(y), detached(y))
    other = i != j
    i, j = i[other], j[other]
    d = y[:, i] - y[:, j]
    g = _spiky(d, h)
    omega = _sum(i, _cross(velocity[:, j] - velocity[:, i], g), n)
    magnitude = _safe_norm(omega)
    eta = _sum(i, (magnitude[j] - magnitude[i]) * g, n)
    length = _safe_norm(eta)
    normal = eta * torch.where(length > 0, 1.0 / torch.where(length > 0, length, torch.ones_like(length)), torch.zeros_like(length))
    confined = velocity + dt * p["vorticity_confinement"] * _cross(normal, omega)
    smooth = _sum(i, _poly6((d * d).sum(0), h) * (confined[:, j] - confined[:, i]), n)
    return y, confined + p["xsph_viscosity"] * smooth


def _cubic(r, h):
    q = r / h
    c = 8.0 / (PI * h ** 3)
    return torch.where(q <= 0.5, c * (6.0 * q ** 3 - 6.0 * q ** 2 + 1.0), 2.0 * c * (1.0 - q) ** 3)


def _cubic_gradient(d, r, h):
    q = r / h
    c = 8.0 / (PI * h ** 3)
    der = torch.where(q <= 0.5, 18.0 * q * q - 12.0 * q, -6.0 * (1.0 - q) ** 2)
    safe = torch.where(r > 0, r, torch.ones_like(r))
    return d * torch.where(r > 0, c * der / (h * safe), torch.zeros_like(r))


def _gradient_norm(h, radius):
    """|sum grad W|^2 + sum |grad W|^2 over a lattice at the particle diameter, a float32 loop by definition."""
    h, step = F32(h), F32(2.0) * F32(radius)
    c = F32(8.0) / (F32(PI) * h * h * h)
    axis, a = [], -h
    while a <= h:
        axis.append(a)
        a = F32(a + step)
    total, squares = np.zeros(3, F32), F32(0.0)
    for x in axis:
        for y in axis:
            for z in axis:
                r2 = x * x + y * y + z * z
                r = F32(np.sqrt(r2))
                if r != 0.0 and r < h:
                    q = r / h
                    der = F32(18.0) * q * q - F32(12.0) * q if q <= 0.5 else F32(-6.0) * (F32(1.0) - q) * (F32(1.0) - q)
                    s = c * der / (h * r)
                    total = total + s * np.array([x, y, z], F32)
                    squares = squares + s * s * r2
    return float((total * total).sum() + squares)


def _sph_substep(x, v, control, p, warm, h, dt, box, radius, method):
    n = x.shape[1]
    mass, rest, visc = p["masses"], p["rest_densities"], p["viscosities"]
    grid = _Pairs(x.detach(), x.detach(), h, box)
    ai, aj = grid.within(x.detach(), x.detach())
    other = ai != aj
    i, j = ai[other], aj[other]
    d = x[:, i] - x[:, j]
    r = _safe_norm(d)
    grad = _cubic_gradient(d, r, h)
    gravity = torch.tensor([0.0, float(F32(-9.8)), 0.0], dtype=x.dtype, device=x.device)[:, None]
    rho = _sum(ai, mass[aj] * _cubic(_safe_norm(x[:, ai] - x[:, aj]), h), n)

    def pressure_acceleration(pressure):
        term = pressure / (rho * rho)
        return _sum(i, grad * (-mass[j] * (term[i] + term[j])), n)

    def predict(a):
        vel = v + dt * a
        pos = x + dt * vel
        lo = float(F32(0.0) + F32(radius))
        hi = torch.tensor([float(F32(b) - F32(radius)) for b in box], dtype=x.dtype, device=x.device)[:, None]
        hit = ((pos < lo) | (pos > hi)).any(0)
        return _clamped(pos, box, radius), torch.where(hit, torch.zeros_like(vel), vel)

    if method == "wcsph":
        c, gamma, tension = p["speed_of_sound"], p["tait_exponent"], p["surface_tensions"]
        pressure = rest * c * c * ((rho / rest) ** gamma - 1.0) / gamma
        approach = ((v[:, i] - v[:, j]) * d).sum(0)
        nu = 2.0 * (0.5 * (visc[i] + visc[j])) * h * (0.5 * (c[i] + c[j])) / (rho[i] + rho[j])
        pi = torch.where(approach < 0, -nu * approach / (r * r + 0.01 * h * h), torch.zeros_like(r))
        diameter = 2.0 * float(F32(radius))
        contact = _cubic(torch.tensor(diameter, dtype=x.dtype, device=x.device), h)
        weight = torch.where(r > diameter, _cubic(r, h), contact)
        a = pressure_acceleration(pressure) + _sum(i, grad * (-mass[j] * pi), n) \
            + _sum(i, d * (-tension[i] * mass[j] * weight / mass[i]), n) + gravity + control
        return predict(a) + ((None, None),)
    lap = 45.0 * (h - r) / (PI * h ** 6)
    base = gravity + control + _sum(i, (v[:, j] - v[:, i]) * (0.5 * (visc[i] + visc[j]) * mass[j] * lap / rho[j]), n)
    norm = _gradient_norm(h, radius)

    def solve(pressure, a, count, extra, relaxation, volume, target):
        for _ in range(count):
            star, _ = predict(base + a + extra)
            si, sj = grid.within(star.detach(), star.detach())
            predicted = _sum(si, mass[sj] * _cubic(_safe_norm(star[:, si] - star[:, sj]), h), n)
            pressure = torch.relu(pressure + relaxation / (2.0 * dt * dt * volume * volume * norm) * (predicted - target))
            a = pressure_acceleration(pressure)
        return pressure, a

    zero = torch.zeros_like(x)
    if method in ("pcisph", "iisph"):
        relaxation = p["pressure_relaxation" if method == "pcisph" else "jacobi_relaxation"]
        volume = mass / (rest if method == "pcisph" else rho)
        _, a = solve(torch.zeros_like(mass), zero, 6, zero, relaxation, volume, rest)
        return predict(base + a) + ((None, None),)
    volume = mass / rho
    first, a = solve(warm[0], pressure_acceleration(warm[0]), 4, zero, p["divergence_relaxation"], volume, rho)
    second, b = solve(warm[1], pressure_acceleration(warm[1]), 6, a, p["density_relaxation"], volume, rest)
    return predict(base + a + b) + ((first, second),)


def exact(case, seed):
    """The pass in 64 bits.  None for rollouts, which amplify any rounding of their first steps, and
    for adjoints whose stored pair terms would not fit the card."""
    kind = case["kind"]
    if kind == "rollout" or (kind in ("grad", "sph_grad") and _particles(case) > 140000):
        return None
    data = _inputs(case, seed)
    wide = lambda t: t.double()
    h, dt = data["h"], data["dt"]
    radius = float(F32(0.2) * F32(h))
    x, v, control = wide(data["x"]), wide(data["v"]), wide(data["control"])
    p = {k: wide(t) for k, t in data["parameters"].items()}
    if kind == "batch":
        xs, vs, first = [], [], 0
        for count, box in zip(data["counts"], data["boxes"]):
            part = slice(first, first + count)
            a, b = _pbf_substep(x[:, part], v[:, part], control[:, part], {k: t[part] for k, t in p.items()}, h, dt, box, radius,
                                case["iterations"], [])
            xs.append(a)
            vs.append(b)
            first += count
        return {"positions": torch.cat(xs, 1), "velocities": torch.cat(vs, 1)}
    box = data["boxes"][0]
    names = _PBF_ADJOINTS if kind == "grad" else _SPH_ADJOINTS.get(case["method"], ())
    leaves = []
    if kind in ("grad", "sph_grad"):
        leaves = [t.requires_grad_(True) for t in (x, v, control)] + [p[name].requires_grad_(True) for name in names]
    with torch.set_grad_enabled(bool(leaves)), torch.autograd.forward_ad.dual_level():
        if kind == "tangent":
            x, v, control = (torch.autograd.forward_ad.make_dual(a, wide(b)) for a, b in zip((x, v, control), data["tangent"]))
        if kind in ("sph", "sph_grad"):
            warm = tuple(wide(t) for t in data["warm"]) if "warm" in data else None
            xo, vo, pressures = _sph_substep(x, v, control, p, warm, h, dt, box, radius, case["method"])
        else:
            xo, vo = _pbf_substep(x, v, control, p, h, dt, box, radius, case["iterations"], data["plates"])
        out = {"positions": xo.detach(), "velocities": vo.detach()}
        if kind == "tangent":
            parts = [torch.autograd.forward_ad.unpack_dual(t) for t in (xo, vo)]
            out = {"positions": parts[0].primal, "velocities": parts[1].primal, "position_tangent": parts[0].tangent,
                   "velocity_tangent": parts[1].tangent}
        if kind == "sph" and case["method"] == "dfsph":
            out["divergence_pressure"], out["density_pressure"] = pressures
        if leaves:
            grads = torch.autograd.grad((xo, vo), leaves, data["adjoint"], allow_unused=True)
            grads = [torch.zeros_like(t) if g is None else g for g, t in zip(grads, leaves)]
            out.update(position_adjoint=grads[0], velocity_adjoint=grads[1], control_adjoint=grads[2])
            out.update({name + "_adjoint": g for name, g in zip(names, grads[3:])})
    if kind == "host":
        out = {k: t.cpu() for k, t in out.items()}
    return out
