"""Performance cases of the rollout engine: the calls that programs make of it, as data.

``listed()`` names the standing cases, ``draw(rng)`` gives further ones of the same ranges,
``prepare(case, seed)`` builds what a program holds before the call, ``run(state)`` is one
pass through the public entry points, ``work(case)`` the bytes and operations that a pass
cannot do without, and ``exact(case, seed)`` the same results in 64 bits from plain torch.

Kinds of call:
  step    ``simulate.step``: one physics step, functional (inputs kept)
  run     ``simulate.run``: a rollout returning its final state
  record  ``simulate.simulate``: a rollout returning its per-step timeseries
  batch   ``Plan.rollout``: uneven rollouts advanced together in place
  grad    ``autodiff.rollout`` and ``torch.autograd.grad``: a rollout and its gradient
  gym     ``BatchedEnv.step``: environments with action, observation and reward
"""
import dataclasses
import math
import random

import numpy as np
import torch

from microcosmos_b200 import autodiff
from microcosmos_b200.config import COSSERAT_SCHEME, PBD_SCHEME, baseline_config
from microcosmos_b200.engine import Actuation, DeviceState, Plan
from microcosmos_b200.gym import BatchedEnv, LineEnv
from microcosmos_b200.simulate import run as simulate_run, simulate, step as simulate_step
from microcosmos_b200.structs import Edges, Fields, Nodes

DT = 0.01
BATCH_SIDES = (128, 192, 256, 384, 512)


def listed():
    return [
        # one functional step of a toy world: an interactive loop, or a user's own control code
        {"name": "step-32", "kind": "step", "config": "baseline", "h": 32, "w": 32, "filaments": 2, "nodes": 12,
         "steps": 1},
        # the small benchmark configuration, as parameter studies run it by the thousand
        {"name": "run-128", "kind": "run", "config": "baseline", "h": 128, "w": 128, "filaments": 4, "nodes": 32,
         "steps": 50},
        # one worm on a 50 x 50 grid with its whole timeseries kept for plots and frames
        {"name": "record-worm-50", "kind": "record", "config": "pbd", "h": 50, "w": 50, "filaments": 1, "nodes": 20,
         "steps": 100},
        # the other rod solver, a 3-point kernel and a ragged domain (not square, mixed factors)
        {"name": "run-ragged-180x300", "kind": "run", "config": "cosserat", "h": 180, "w": 300, "filaments": 12,
         "nodes": 41, "steps": 40},
        # the method at scale: one large swarm
        {"name": "run-1024", "kind": "run", "config": "baseline", "h": 1024, "w": 1024, "filaments": 256, "nodes": 64,
         "steps": 16},
        # the largest single lattice, populations larger than the cache
        {"name": "run-2048", "kind": "run", "config": "baseline", "h": 2048, "w": 2048, "filaments": 512, "nodes": 64,
         "steps": 8},
        # a part and the whole of an evolutionary search's population, and a serving epoch
        {"name": "batch-64", "kind": "batch", "config": "baseline", "rollouts": 64, "steps": 10},
        {"name": "batch-256", "kind": "batch", "config": "baseline", "rollouts": 256, "steps": 4},
        # differentiation: the benchmark's swimmer problem, and a larger served request
        {"name": "grad-256", "kind": "grad", "config": "baseline", "h": 256, "w": 256, "filaments": 8, "nodes": 48,
         "steps": 48},
        {"name": "grad-640", "kind": "grad", "config": "baseline", "h": 640, "w": 640, "filaments": 64, "nodes": 64,
         "steps": 12},
        # reinforcement learning: a population of environments stepped together
        {"name": "gym-256", "kind": "gym", "config": "pbd", "h": 128, "w": 128, "filaments": 1, "nodes": 16,
         "envs": 256, "steps": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "run", "run", "record", "batch", "grad", "gym"])
    if kind == "batch":
        return {"kind": kind, "config": "baseline", "rollouts": _log_int(rng, 2, 200), "steps": rng.randint(2, 8)}
    nodes = _log_int(rng, 12, 128)
    if kind == "gym":
        side = rng.choice([64, 96, 128])
        return {"kind": kind, "config": "pbd", "h": side, "w": rng.choice([64, 96, 128]), "filaments": 1,
                "nodes": min(nodes, 24), "envs": _log_int(rng, 2, 256), "steps": rng.randint(2, 8)}
    # sides of every parity and factor; a domain need not be square
    top = {"step": 256, "run": 1200, "record": 256, "grad": 512}[kind]
    h = _log_int(rng, 56, top)
    w = h if rng.random() < 0.4 else max(56, min(top, int(h * rng.uniform(0.6, 1.6))))
    if rng.random() < 0.5:
        h, w = (max(64, v // 32 * 32) for v in (h, w))
    filaments = _log_int(rng, 1, max(1, min(256, h * w // (64 * nodes))))
    steps = {"step": 1, "run": rng.randint(4, 24), "record": rng.randint(8, 40), "grad": rng.randint(4, 16)}[kind]
    return {"kind": kind, "config": rng.choice(["baseline", "baseline", "pbd", "cosserat"]), "h": h, "w": w,
            "filaments": filaments, "nodes": nodes, "steps": steps}


# ---------------------------------------------------------------- inputs
def _config(name):
    if name == "baseline":  # 4-point kernel, steric field on
        return baseline_config()
    if name == "cosserat":  # the implicit rod solver, 3-point kernel, steric field on
        return dataclasses.replace(COSSERAT_SCHEME, enable_steric=True, ibm_kernel_size=3)
    return PBD_SCHEME  # the gym default: 2-point kernel, no steric field


def _rods(rng, h, w, filaments, n):
    """Straight rods of unit spacing at uniform places and angles, with curvature waves: numpy
    arrays as a program builds them."""
    F = filaments
    first = np.arange(F)[:, None] * n
    pairs = np.stack([first + np.arange(n - 1), first + np.arange(1, n)], -1).reshape(-1, 2).astype(np.int32)
    e0 = np.arange(F)[:, None] * (n - 1)
    bends = np.stack([e0 + np.arange(n - 2), e0 + np.arange(1, n - 1)], -1).reshape(-1, 2).astype(np.int32)
    centre = rng.uniform(0, 1, (F, 1, 2)) * np.array([w, h])
    angle = rng.uniform(0, 2 * np.pi, (F, 1))
    along = np.arange(n) - (n - 1) / 2
    pos = centre + np.stack([along * np.cos(angle), along * np.sin(angle)], -1)
    pos = np.mod(pos.reshape(-1, 2).astype(np.float32), np.array([w, h], np.float32)).astype(np.float32)
    size = np.array([w, h], np.float32)
    d = np.mod(pos[pairs[:, 1]] - pos[pairs[:, 0]] + size / 2, size) - size / 2
    amp = np.repeat(rng.uniform(0.1, 0.3, F), n - 2)
    omega = np.repeat(2 * np.pi / rng.uniform(100, 400, F), n - 2)
    phase = np.tile(-2 * np.pi * np.arange(n - 2) / max(n - 2, 1), F) + np.repeat(rng.uniform(0, 2 * np.pi, F), n - 2)
    f32 = lambda a: np.ascontiguousarray(a, dtype=np.float32)  # noqa: E731
    return {"pos": pos, "pairs": pairs, "bends": bends, "theta": f32(np.arctan2(d[:, 1], d[:, 0])),
            "rest": np.ones(len(pairs), np.float32), "kb": np.full(len(bends), 0.1, np.float32),
            "angles": f32(amp * np.sin(phase)),
            "act": (np.zeros(len(bends), np.float32), f32(amp), f32(omega), f32(phase))}


_E = ((0, 0), (1, 0), (0, 1), (-1, 0), (0, -1), (1, 1), (-1, 1), (-1, -1), (1, -1))
_WEIGHTS = (4 / 9,) + (1 / 9,) * 4 + (1 / 36,) * 4


def _populations(h, w, seed, device):
    """Equilibrium populations of a fluid at rest but for a velocity noise of 1e-3."""
    g = torch.Generator(device=device).manual_seed(seed)
    u = torch.randn((2, h, w), generator=g, device=device) * 1e-3
    usq = u[0] * u[0] + u[1] * u[1]
    f = torch.empty((9, h, w), device=device)
    for i, (ex, ey) in enumerate(_E):
        eu = ex * u[0] + ey * u[1]
        f[i] = _WEIGHTS[i] * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * usq)
    return f


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _world(case, seed):
    rods = _rods(np.random.default_rng(seed), case["h"], case["w"], case["filaments"], case["nodes"])
    return rods, _populations(case["h"], case["w"], seed, _device())


def _population_sizes(case, seed):
    """(side, filaments, nodes) of each rollout of a batch: fixed by the case, so that another
    seed changes the places and not the amount of work."""
    r = random.Random(case["rollouts"])
    return [(r.choice(BATCH_SIDES), r.randint(1, 32), r.randint(16, 128)) for _ in range(case["rollouts"])]


def _batch_parts(case, seed):
    parts = []
    for i, (side, filaments, nodes) in enumerate(_population_sizes(case, seed)):
        rods = _rods(np.random.default_rng([seed, i]), side, side, filaments, nodes)
        parts.append((side, rods, _populations(side, side, seed * 1000 + i, _device())))
    return parts


def _actions(case, seed):
    g = torch.Generator(device=_device()).manual_seed(seed)
    B, n = case["envs"], case["nodes"]
    return [{"d_rest_length": 0.1 * torch.randn((B, n - 1), generator=g, device=_device()),
             "d_bending_angle": 0.2 * torch.randn((B, n - 2), generator=g, device=_device())}
            for _ in range(case["steps"])]


def prepare(case, seed):
    cfg = _config(case["config"])
    kind, steps = case["kind"], case["steps"]
    if kind == "gym":
        env = LineEnv(num_nodes=case["nodes"], grid_shape=(case["h"], case["w"]), energy_amplitude=1.0,
                      max_steps=10 ** 9)
        batch = BatchedEnv(env, case["envs"])
        _, state = batch.reset(list(range(case["envs"])))
        return {"kind": kind, "batch": batch, "state": state, "actions": _actions(case, seed)}
    if kind == "batch":
        parts = _batch_parts(case, seed)
        # a population's results are read together: the states are views of one buffer per array
        flat = {k: [] for k in ("pos", "theta", "f")}
        for side, rods, f in parts:
            flat["pos"].append(rods["pos"].reshape(-1))
            flat["theta"].append(rods["theta"])
            flat["f"].append(f.reshape(-1))
        pos = torch.as_tensor(np.concatenate(flat["pos"]), device="cuda")
        vel = torch.zeros_like(pos)
        theta = torch.as_tensor(np.concatenate(flat["theta"]), device="cuda")
        f = torch.cat(flat["f"])
        cells = f.numel() // 9
        steric, u = torch.zeros(cells, device="cuda"), torch.zeros(2 * cells, device="cuda")
        states, acts, at_n, at_e, at_c = [], [], 0, 0, 0
        for side, rods, _ in parts:
            N, E, C = len(rods["pos"]), len(rods["pairs"]), side * side
            dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
            states.append(DeviceState(
                H=side, W=side, position=pos[2 * at_n:2 * (at_n + N)].view(N, 2),
                velocity=vel[2 * at_n:2 * (at_n + N)].view(N, 2), theta=theta[at_e:at_e + E],
                rest_lengths=dev(rods["rest"]), bending_rest_angles=dev(rods["angles"]),
                bending_stiffness=dev(rods["kb"]), steric=steric[at_c:at_c + C].view(side, side),
                fluid_velocity=u[2 * at_c:2 * (at_c + C)].view(2, side, side),
                f_grid=f[9 * at_c:9 * (at_c + C)].view(9, side, side), pairs=rods["pairs"],
                bending_pairs=rods["bends"]))
            acts.append(Actuation(*[dev(a) for a in rods["act"]]))
            at_n, at_e, at_c = at_n + N, at_e + E, at_c + C
        n = len(states)
        return {"kind": kind, "plan": Plan.for_states(states, [cfg] * n, [DT] * n), "states": states, "acts": acts,
                "steps": steps, "out": {"position": pos, "velocity": vel, "theta": theta, "f_grid": f,
                                        "steric": steric, "fluid_velocity": u}}
    rods, f = _world(case, seed)
    dev = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    if kind == "grad":
        leaves = {"position": dev(rods["pos"]), "velocity": torch.zeros((len(rods["pos"]), 2), device="cuda"),
                  "theta": dev(rods["theta"]), "f_grid": f, "c": dev(rods["act"][0]), "amp": dev(rods["act"][1]),
                  "phase": dev(rods["act"][3])}
        for t in leaves.values():
            t.requires_grad_(True)
        return {"kind": kind, "leaves": leaves, "omega": dev(rods["act"][2]), "rest": dev(rods["rest"]),
                "kb": dev(rods["kb"]), "angles": dev(rods["angles"]), "pairs": rods["pairs"], "bends": rods["bends"],
                "cfg": cfg, "steps": steps}
    N = len(rods["pos"])
    nodes = Nodes(position=dev(rods["pos"]), velocity=torch.zeros((N, 2), device="cuda"),
                  color_bend=torch.zeros(N, dtype=torch.int32, device="cuda"),
                  debug_vector=torch.zeros((N, 2), device="cuda"))
    edges = Edges(pairs=rods["pairs"], theta=dev(rods["theta"]), rest_lengths=dev(rods["rest"]),
                  bending_pairs=rods["bends"], bending_rest_angles=dev(rods["angles"]),
                  bending_stiffness=dev(rods["kb"]))
    h, w = case["h"], case["w"]
    fields = Fields(grid_shape=(h, w), steric=torch.zeros((h, w), device="cuda"),
                    fluid_velocity=torch.zeros((2, h, w), device="cuda"), f_grid=f)
    return {"kind": kind, "nodes": nodes, "edges": edges, "fields": fields, "cfg": cfg, "steps": steps,
            "act": tuple(dev(a) for a in rods["act"])}


# ---------------------------------------------------------------- one pass
def _state_out(nodes, edges, fields):
    return {"position": nodes.position, "velocity": nodes.velocity, "theta": edges.theta, "f_grid": fields.f_grid,
            "steric": fields.steric, "fluid_velocity": fields.fluid_velocity}


def run(state):
    kind = state["kind"]
    if kind == "step":
        return _state_out(*simulate_step(state["nodes"], state["edges"], state["fields"], DT, state["cfg"]))
    if kind == "run":
        return _state_out(*simulate_run(state["nodes"], state["edges"], state["fields"], DT, state["steps"],
                                        state["cfg"], actuation=state["act"]))
    if kind == "record":
        nodes, fields = simulate(state["nodes"], state["edges"], state["fields"], DT, state["steps"],
                                          state["cfg"], actuation=state["act"])
        return {"position": nodes.position, "velocity": nodes.velocity, "steric": fields.steric,
                "fluid_velocity": fields.fluid_velocity}
    if kind == "batch":
        state["plan"].rollout(state["states"], state["steps"], actuations=state["acts"])
        return state["out"]
    if kind == "grad":
        v = state["leaves"]
        out = autodiff.rollout(v["position"], v["velocity"], v["theta"], v["f_grid"], state["rest"], state["kb"],
                               state["angles"], state["pairs"], state["bends"], state["cfg"], DT, state["steps"],
                               actuation=(v["c"], v["amp"], state["omega"], v["phase"]))
        loss = (out[0][:, 0] - v["position"][:, 0]).mean()  # centre-of-mass displacement
        grads = torch.autograd.grad(loss, list(v.values()))
        return {"loss": loss.detach(), "position": out[0].detach(), "f_grid": out[3].detach(),
                "grads": dict(zip(v, grads))}
    outs = []
    for action in state["actions"]:
        obs, _, reward, _, _ = state["batch"].step(None, state["state"], action)
        outs.append({"observation": obs, "reward": reward})
    return outs


# ---------------------------------------------------------------- work
def work(case):
    cfg = _config(case["config"])
    if case["kind"] == "batch":
        parts = [(s * s, F * n) for s, F, n in _population_sizes(case, 0)]
    elif case["kind"] == "gym":
        parts = [(case["h"] * case["w"], case["nodes"])] * case["envs"]
    else:
        parts = [(case["h"] * case["w"], case["filaments"] * case["nodes"])]
    cells, nodes, steps = sum(p[0] for p in parts), sum(p[1] for p in parts), case["steps"]
    k2 = cfg.ibm_kernel_size ** 2
    steric = cfg.enable_steric
    # a step: nine populations read and written per cell, the steric field written; per node its
    # position, velocity, angle, rest state and actuation read, and the first three written
    bytes_step = cells * (72 + (4 if steric else 0)) + nodes * 56
    # TRT collision about 200 a cell, the separable filter's transforms, rod iterations, stencil
    # weights and the forcing rounds' interpolation and spreading
    flops_step = (cells * (200 + (100 if steric else 0)) + nodes * (cfg.cycles_per_step * 60 + 150)
                  + nodes * k2 * (20 + 8 * cfg.ibm_iterations))
    if case["kind"] == "record":
        bytes_step += cells * 12 + nodes * 16  # the recorded fields and nodes
    if case["kind"] == "grad":
        # the forward step, its recomputation from a checkpoint, and the reverse step: the
        # cotangents of the populations read and written beside the step's input
        bytes_step += cells * (72 + 108) + nodes * 168
        flops_step *= 4
    return {"bytes": float(bytes_step * steps), "flops": float(flops_step * steps)}


# ---------------------------------------------------------------- the same in 64 bits
_EPS = float(np.finfo(np.float32).eps)


def _scale_clamp(x, y, vmax):
    return torch.clamp(vmax / (torch.sqrt(x * x + y * y + _EPS) + _EPS), max=1.0) if not x.requires_grad else \
        torch.minimum(torch.ones_like(x), vmax / (torch.sqrt(x * x + y * y + _EPS) + _EPS))


def _add_at(size, index, values):
    """(B, size) zeros with values (B, M) added at index (M,) or (B, M)."""
    out = torch.zeros(values.shape[0], size, dtype=values.dtype, device=values.device)
    return out.scatter_add(1, index.expand(values.shape[0], -1), values)


def _steric64(cfg, pred, h, w):
    size = torch.tensor([w, h], dtype=torch.float64, device=pred.device)
    p = torch.remainder(pred, size)
    base = torch.floor(p.detach())
    t = p - base
    x0, y0 = torch.remainder(base[..., 0].long(), w), torch.remainder(base[..., 1].long(), h)
    x1, y1 = (x0 + 1) % w, (y0 + 1) % h
    dx, dy = t[..., 0], t[..., 1]
    index = torch.cat([y0 * w + x0, y0 * w + x1, y1 * w + x0, y1 * w + x1], 1)
    weight = torch.cat([(1 - dx) * (1 - dy), dx * (1 - dy), (1 - dx) * dy, dx * dy], 1) * cfg.steric_scatter_value
    rho = _add_at(h * w, index, weight).view(-1, h, w)
    fy, fx = (torch.fft.fftfreq(n, dtype=torch.float64, device=pred.device) for n in (h, w))
    kf = torch.exp(-2 * math.pi ** 2 * cfg.steric_sigma ** 2 * (fy[:, None] ** 2 + fx[None, :] ** 2))
    V = torch.fft.ifft2(torch.fft.fft2(rho) * kf).real
    flat = V.reshape(-1, h * w)

    def sample(yy, xx):
        ly, lx = torch.floor(yy.detach()), torch.floor(xx.detach())
        ty, tx = yy - ly, xx - lx
        iy, ix = ly.long(), lx.long()
        out = 0
        for a, wy in ((0, 1 - ty), (1, ty)):
            for b, wx in ((0, 1 - tx), (1, tx)):
                out = out + wy * wx * flat.gather(1, torch.remainder(iy + a, h) * w + torch.remainder(ix + b, w))
        return out

    x, y = p[..., 0], p[..., 1]
    force = -torch.stack([sample(y, x + 0.5) - sample(y, x - 0.5), sample(y + 0.5, x) - sample(y - 0.5, x)], -1)
    N, s2 = p.shape[1], cfg.steric_sigma ** 2
    near = torch.zeros_like(force)
    for o in range(-cfg.steric_neighbor_skip, cfg.steric_neighbor_skip + 1):
        j = torch.arange(N, device=p.device) + o
        ok = ((j >= 0) & (j < N)).double()[None, :, None]
        r = torch.remainder(p - p[:, j.clamp(0, N - 1)] + size / 2, size) - size / 2
        near = near + ok * r * torch.exp(-(r * r).sum(-1, keepdim=True) / (2 * s2)) / (2 * math.pi * s2)
    return V, force - cfg.steric_scatter_value / s2 * near


def _step64(cfg, s, angles):
    """One step of B worlds of one topology; s: a dict of (B, ...) float64 tensors, "pairs", "bends"."""
    pos0, h, w = s["pos"], s["f"].shape[2], s["f"].shape[3]
    B, N = pos0.shape[:2]
    dev = pos0.device
    size = torch.tensor([w, h], dtype=torch.float64, device=dev)
    image = lambda d: torch.remainder(d + size / 2, size) - size / 2  # noqa: E731
    src, tgt, ein, eout = s["pairs"][:, 0], s["pairs"][:, 1], s["bends"][:, 0], s["bends"][:, 1]
    E = src.numel()
    ones = lambda idx, n: _add_at(n, idx, torch.ones(1, idx.numel(), dtype=torch.float64, device=dev))  # noqa: E731
    edeg = (ones(ein, E) + ones(eout, E)).clamp(min=1)
    ndeg = (ones(src, N) + ones(tgt, N)).clamp(min=1)[..., None]
    theta, rest, kb = s["theta"], s["rest"], s["kb"]
    pos = pos0 + s["vel"] * cfg.damping * DT
    steric = s["steric"]
    if cfg.enable_steric:
        steric, force = _steric64(cfg, pos, h, w)
        pos = pos + force * cfg.steric_strength * DT
    start = pos
    wrap = lambda a: torch.remainder(a + math.pi, 2 * math.pi) - math.pi  # noqa: E731
    both = lambda v: torch.zeros(B, N, 2, dtype=torch.float64, device=dev).index_add(1, src, v).index_add(  # noqa: E731
        1, tgt, -v)
    for _ in range(cfg.cycles_per_step):
        corr = (wrap(theta[:, eout] - theta[:, ein]) - angles) * kb * 0.5
        turn = torch.zeros_like(theta).index_add(1, ein, corr).index_add(1, eout, -corr) / edeg
        seg = image(pos[:, tgt] - pos[:, src])
        if cfg.solver_type == "cosserat":
            theta = theta + turn
            theta = theta + wrap(torch.atan2(seg[..., 1], seg[..., 0]) - theta) * 0.05
            d = torch.stack([torch.cos(theta), torch.sin(theta)], -1)
            ks, inertia = cfg.stiffness_stretch, 1.0 / cfg.dt ** 2
            hess = ks / (rest * rest)
            den = inertia + torch.zeros(B, N, dtype=torch.float64, device=dev).index_add(1, src, hess).index_add(
                1, tgt, hess)
            pull = both((ks / rest)[..., None] * (seg / rest[..., None] - d))
            pos = pos + (inertia * (start - pos) + pull) / den[..., None]
        else:
            theta = theta + turn * 1.8
            d = torch.stack([torch.cos(theta), torch.sin(theta)], -1)
            L = torch.sqrt((seg * seg).sum(-1, keepdim=True))
            stretch = seg / torch.clamp(L, min=1e-8) * (L - rest[..., None])
            shear = (seg - d * rest[..., None]) - stretch
            pos = pos + both((stretch + shear * cfg.stiffness_shear) * cfg.stiffness_stretch * 0.5) / ndeg
    vel = (pos - pos0) / DT
    # immersed boundary (scale: lattice over domain, the axes in the order that the engine documents)
    scale = torch.tensor([w / h, h / w], dtype=torch.float64, device=dev)
    vmax = cfg.max_fluid_velocity * 0.5 * (w / h + h / w)
    point = (pos * scale).detach()
    K = cfg.ibm_kernel_size
    corner = torch.floor(point) - (K - 1) // 2
    offs = torch.arange(K, device=dev)
    cell = corner[..., None] + offs  # (B, N, 2, K)
    r = (cell - point[..., None]).abs() / (K / 2)
    phi = torch.where(r <= 2, 0.25 * (1 + torch.cos(math.pi * r / 2)), torch.zeros_like(r))
    wts = (phi[:, :, 0, :, None] * phi[:, :, 1, None, :]).reshape(B, N, K * K)
    wts = wts / (wts.sum(-1, keepdim=True) + _EPS)
    cx, cy = torch.remainder(cell[:, :, 0].long(), w), torch.remainder(cell[:, :, 1].long(), h)
    flat = (cy[:, :, None, :] * w + cx[:, :, :, None]).reshape(B, N * K * K)
    wf = wts.reshape(B, -1)
    f = torch.maximum(s["f"], torch.full((), _EPS, dtype=torch.float64, device=dev)).reshape(B, 9, h * w)
    rho = torch.maximum(f.sum(1), torch.full((), 0.1, dtype=torch.float64, device=dev))
    e = torch.tensor(_E, dtype=torch.float64, device=dev)
    ux, uy = ((f * e[:, k].view(1, 9, 1)).sum(1) / rho for k in (0, 1))
    c = _scale_clamp(ux, uy, vmax)
    ux, uy = ux * c, uy * c
    inv = 1 / _add_at(h * w, flat, wf).clamp(min=1)
    gx, gy = ux, uy
    node = vel * scale * DT
    at = lambda field: (field.gather(1, flat).view(B, N, K * K) * wts).sum(-1)  # noqa: E731
    for _ in range(cfg.ibm_iterations):
        sx, sy = (node[..., 0] - at(gx)) * cfg.ibm_relaxation, (node[..., 1] - at(gy)) * cfg.ibm_relaxation
        c = _scale_clamp(sx, sy, vmax)
        spread = lambda v: _add_at(h * w, flat, ((v * c)[..., None] * wts).reshape(B, -1)) * inv  # noqa: E731
        gx, gy = gx + spread(sx), gy + spread(sy)
    c = _scale_clamp(gx, gy, vmax)
    Fx, Fy = (gx * c - ux) * rho, (gy * c - uy) * rho
    wp = min(max(1 / (3 * cfg.viscosity + 0.5), 0.0), 1.9)
    wm = 1 / (cfg.lambda_trt / max(1 / max(wp, _EPS) - 0.5, _EPS) + 0.5)
    vx, vy = ux + 0.5 * Fx / rho, uy + 0.5 * Fy / rho
    wi = torch.tensor(_WEIGHTS, dtype=torch.float64, device=dev).view(1, 9, 1)
    ev = e[:, 0].view(1, 9, 1) * vx[:, None] + e[:, 1].view(1, 9, 1) * vy[:, None]
    eF = e[:, 0].view(1, 9, 1) * Fx[:, None] + e[:, 1].view(1, 9, 1) * Fy[:, None]
    feq = rho[:, None] * wi * (1 + 3 * ev + 4.5 * ev * ev - 1.5 * (vx * vx + vy * vy)[:, None])
    src_f = wi * (3 * (eF - (vx * Fx + vy * Fy)[:, None]) + 9 * ev * eF)
    opp = [0, 3, 4, 1, 2, 7, 8, 5, 6]
    even = lambda a: 0.5 * (a + a[:, opp])  # noqa: E731
    odd = lambda a: 0.5 * (a - a[:, opp])  # noqa: E731
    post = (f - wp * (even(f) - even(feq)) - wm * (odd(f) - odd(feq)) + (1 - 0.5 * wp) * even(src_f)
            + (1 - 0.5 * wm) * odd(src_f))
    post = torch.maximum(post, torch.full((), _EPS, dtype=torch.float64, device=dev)).view(B, 9, h, w)
    f_new = torch.stack([torch.roll(post[:, i], (ey, ex), (1, 2)) for i, (ex, ey) in enumerate(_E)], 1)
    react = torch.stack([at(Fx), at(Fy)], -1)
    vel = vel - react / cfg.node_mass / (scale * DT)
    return dict(s, pos=torch.remainder(pos, size), vel=vel, theta=theta, f=f_new, steric=steric,
                u=torch.stack([vx, vy], 1).view(B, 2, h, w))


def _world64(rods, f):
    dev = f.device
    up = lambda a: torch.as_tensor(a, device=dev).double()[None]  # noqa: E731
    return {"pos": up(rods["pos"]), "vel": torch.zeros_like(up(rods["pos"])), "theta": up(rods["theta"]),
            "rest": up(rods["rest"]), "kb": up(rods["kb"]), "f": f.double()[None],
            "steric": torch.zeros((1,) + tuple(f.shape[1:]), dtype=torch.float64, device=dev), "u": None,
            "pairs": torch.as_tensor(rods["pairs"], device=dev).long(),
            "bends": torch.as_tensor(rods["bends"], device=dev).long()}


def _angles64(act, t):
    c, amp, omega, phase = act
    return (c + amp * torch.sin(omega * t + phase))[None]


def _out64(s):
    return {"position": s["pos"][0], "velocity": s["vel"][0], "theta": s["theta"][0], "f_grid": s["f"][0],
            "steric": s["steric"][0], "fluid_velocity": s["u"][0]}


def exact(case, seed):
    cfg, kind = _config(case["config"]), case["kind"]
    dev = _device()
    if kind == "gym":
        B, n, h, w = case["envs"], case["nodes"], case["h"], case["w"]
        xs = np.linspace(w / 2 - (n - 1), w / 2 + (n - 1), n).astype(np.float32)  # spacing 2
        rods = {"pos": np.stack([xs, np.full(n, h / 2, np.float32)], 1), "theta": np.zeros(n - 1, np.float32),
                "rest": np.full(n - 1, 2.0, np.float32), "kb": np.full(n - 2, 0.5, np.float32),
                "pairs": np.stack([np.arange(n - 1), np.arange(1, n)], 1),
                "bends": np.stack([np.arange(n - 2), np.arange(1, n - 1)], 1)}
        f = torch.tensor(_WEIGHTS, device=dev).view(9, 1, 1).expand(9, h, w)
        s = {k: v.expand(B, *v.shape[1:]).clone() if torch.is_tensor(v) and k not in ("pairs", "bends") else v
             for k, v in _world64(rods, f).items()}
        rest, outs = s["rest"], []
        size = torch.tensor([w, h], dtype=torch.float64, device=dev)
        for a in _actions(case, seed):
            s = _step64(cfg, dict(s, rest=rest + a["d_rest_length"].double()), a["d_bending_angle"].double())
            d = torch.remainder(s["pos"] - 30.0 + size / 2, size) - size / 2  # the source at twice its size, 15
            energy = torch.exp(-(d * d).sum(-1) / (2 * 15.0 ** 2))
            centred = s["pos"] - s["pos"].mean(1, keepdim=True)
            outs.append({"observation": torch.cat([centred.reshape(B, -1), s["vel"].reshape(B, -1), energy], 1),
                         "reward": energy.sum(1)})
        return outs
    if kind == "batch":
        done = []
        for side, rods, f in _batch_parts(case, seed):
            s = _world64(rods, f)
            act = [torch.as_tensor(a, device=dev).double() for a in rods["act"]]
            for t in range(case["steps"]):
                s = _step64(cfg, s, _angles64(act, t))
            done.append(_out64(s))
        return {k: torch.cat([o[k].reshape(-1) for o in done]) for k in done[0]}
    rods, f = _world(case, seed)
    act = [torch.as_tensor(a, device=dev).double() for a in rods["act"]]
    s = _world64(rods, f)
    if kind == "step":
        return _out64(_step64(cfg, s, torch.as_tensor(rods["angles"], device=dev).double()[None]))
    if kind == "grad":
        v = {"position": s["pos"], "velocity": s["vel"], "theta": s["theta"], "f_grid": s["f"], "c": act[0],
             "amp": act[1], "phase": act[3]}
        for t in v.values():
            t.requires_grad_(True)
        for t in range(case["steps"]):
            s = _step64(cfg, s, _angles64(act, t))
        loss = (s["pos"][0, :, 0] - v["position"][0, :, 0]).mean()
        grads = torch.autograd.grad(loss, list(v.values()))
        return {"loss": loss.detach(), "position": s["pos"][0].detach(), "f_grid": s["f"][0].detach(),
                "grads": {k: (g if k in ("c", "amp", "phase") else g[0]) for k, g in zip(v, grads)}}
    series = []
    for t in range(case["steps"]):
        s = _step64(cfg, s, _angles64(act, t))
        if kind == "record":
            series.append({k: v for k, v in _out64(s).items() if k not in ("theta", "f_grid")})
    if kind == "record":
        return {k: torch.stack([o[k] for o in series]) for k in series[0]}
    return _out64(s)
