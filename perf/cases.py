"""The work that programs built on this package ask of it, case by case.

A case is a dict of plain values.  ``listed`` gives the fixed ones, ``draw``
one more from the same ranges, ``prepare`` what a program holds before the
call (inputs on the GPU, made from the seed alone, and the simulator, decoder
or network it keeps), ``run`` one pass through the public entry points,
``work`` the bytes and operations a pass cannot do without, and ``exact`` the
pass's outputs in float64 PyTorch, without this package's kernels.

Particles fill a column as in ``scenarios``; they are strained by a few
percent (a settling column), partly yielding, and moving.  They come in cell
order, as the particles of a running simulation do.
"""
import math

import torch
from torch.utils.checkpoint import checkpoint

from reduced_mpm_stress_training_gb300 import MPM_Simulator_WARP
from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300.adjoint import SandRollout, rollout
from reduced_mpm_stress_training_gb300.batched import BatchedMPM
from reduced_mpm_stress_training_gb300.decoder import StressDecoder
from reduced_mpm_stress_training_gb300.scenarios import Scene, batch_64
from reduced_mpm_stress_training_gb300.surrogate import StressMLP, W_COUNT

DEV = "cuda:0"
NU = 0.3
GRAVITY = (0.0, 0.0, -9.8)
MATERIAL = {  # Young's modulus, density, time step
    "sand": (2e5, 2200.0, 5e-5),
    "metal": (1e7, 2700.0, 5e-5),
    "jelly": (1e5, 1000.0, 1e-4),
}
YIELD = 1e5
PHI = 30.0


# --------------------------------------------------------------------------- cases
def listed():
    return [
        # The learned-stress loop on a small object: every step takes u, v and stress
        # from a model and hands the state back (the smallest calls).
        {"name": "loop_jelly_2k", "kind": "loop", "n": 2000, "grid": 32, "material": "jelly", "steps": 4},
        # A small scene stepped by one CUDA graph replay between two frames.
        {"name": "graph_sand_4k", "kind": "graph", "n": 4096, "grid": 32, "material": "sand", "steps": 32},
        # One output frame of the 32k column, stepped call by call.
        {"name": "frame_sand_32k", "kind": "frame", "n": 32768, "grid": 64, "material": "sand", "steps": 20},
        # An odd-sized hardening metal block on the 96^3 grid.
        {"name": "frame_metal_300k", "kind": "frame", "n": 300007, "grid": 96, "material": "metal", "steps": 8},
        # The 1M column of the headline benchmark.
        {"name": "frame_sand_1m", "kind": "frame", "n": 1048576, "grid": 128, "material": "sand", "steps": 8},
        # A production-size column on a 256^3 grid (the largest).
        {"name": "frame_sand_8m", "kind": "frame", "n": 8388608, "grid": 256, "material": "sand", "steps": 4},
        # 64 uneven sand and metal scenes in one engine.
        {"name": "batch_64", "kind": "batch", "scenes": 64, "steps": 4},
        # The reduced sampled-quadrature substep: dense grids around 4,096 sample points.
        {"name": "reduced_sand_1m", "kind": "reduced", "n": 1048576, "grid": 128, "material": "sand", "samples": 4096},
        # The stress decoder (width 30, the reference's default) feeding 1M particles.
        {"name": "decoder_1m", "kind": "decoder", "n": 1048576, "grid": 128, "scale": 10, "label": 6, "siren": False},
        # Gradients of a rollout with respect to v0, E and the friction angle.
        {"name": "grad_sand_131k", "kind": "grad", "n": 131072, "grid": 96, "steps": 10, "every": 5},
        # One training step of the stress network at its batch size.
        {"name": "train_65k", "kind": "train", "rows": 65536},
        # The stress network evaluated on a million strains.
        {"name": "network_1m", "kind": "network", "rows": 1048576},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop", "graph", "frame", "frame", "frame", "batch", "reduced", "decoder", "grad", "train",
                       "network"])
    material = rng.choice(["sand", "sand", "metal", "jelly"])
    if kind in ("loop", "graph"):
        n = _log(rng, 1000, 100000)
        steps = rng.randint(2, 6) if kind == "loop" else 2 * rng.randint(2, 20)
        return {"kind": kind, "n": n, "grid": rng.randint(28, 72), "material": material, "steps": steps}
    if kind == "frame":
        n = _log(rng, 2000, 4000000)
        # one to twelve particles a cell of the column
        grid = int(min(256, max(24, round((n / (0.072 * rng.uniform(1.0, 12.0))) ** (1.0 / 3.0)))))
        return {"kind": kind, "n": n, "grid": grid, "material": material, "steps": rng.randint(2, 20) if n < 300000 else 4}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randint(2, 64), "steps": rng.randint(2, 8)}
    if kind == "reduced":
        n = _log(rng, 3000, 2000000)
        grid = int(min(160, max(24, round((n / (0.072 * rng.uniform(2.0, 10.0))) ** (1.0 / 3.0)))))
        return {"kind": kind, "n": n, "grid": grid, "material": material, "samples": _log(rng, 16, 8192)}
    if kind == "decoder":
        return {"kind": kind, "n": _log(rng, 1000, 2000000), "grid": 64, "scale": rng.choice([5, 8, 10, 10]),
                "label": rng.randint(2, 12), "siren": rng.random() < 0.25}
    if kind == "grad":
        every = rng.randint(2, 5)
        return {"kind": kind, "n": _log(rng, 3000, 200000), "grid": rng.randint(32, 96), "steps": every * rng.randint(1, 2),
                "every": every}
    return {"kind": kind, "rows": _log(rng, 500, 150000) if kind == "train" else _log(rng, 1000, 2000000)}


# --------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _box(grid):
    return ((0.35, 0.35, 0.15), (0.65, 0.65, 0.75)) if grid < 48 else ((0.35, 0.35, 0.05), (0.65, 0.65, 0.85))


def _floor(grid):
    return _box(grid)[0][2]


def _lame(E):
    return E / 2.0 / (1.0 + NU), E * NU / (1.0 + NU) / (1.0 - 2.0 * NU)


def _alpha(phi):
    s = math.sin(phi / 180.0 * 3.14159265)
    return math.sqrt(2.0 / 3.0) * 2.0 * s / (3.0 - s)


def _material(case):
    E, rho, dt = MATERIAL[case.get("material", "sand")]
    mu, lam = _lame(E)
    return {"material": case.get("material", "sand"), "mu": mu, "lam": lam, "alpha": _alpha(PHI), "xi": 0.1,
            "rho": rho, "dt": dt, "E": E}


def _particles(n, grid, mat, g, box=None):
    """float32 particle arrays on the GPU: x0, u, v, C, F, stress (of F), vol, mass, yield."""
    lo, hi = (torch.tensor(b, device=DEV) for b in (box or _box(grid)))
    x = lo + (hi - lo) * torch.rand(n, 3, generator=g, device=DEV)
    c = (x * grid - 0.5).to(torch.int64)  # cell order: 4x4x4 blocks, cells inside a block
    b, i = c // 4, c % 4
    nb = (grid + 3) // 4
    key = ((b[:, 0] * nb + b[:, 1]) * nb + b[:, 2]) * 64 + (i[:, 0] * 4 + i[:, 1]) * 4 + i[:, 2]
    x = x[key.argsort()].contiguous()
    phase = 6.2831853 * torch.rand(3, generator=g, device=DEV)
    wave = torch.sin(9.0 * x[:, [1, 2, 0]] + phase)
    u = 0.001 * wave
    v = 0.3 * wave + 0.02 * torch.randn(n, 3, generator=g, device=DEV)
    v[:, 2] -= 0.5
    C = 1.0 * torch.randn(n, 3, 3, generator=g, device=DEV)
    depth = (hi[2] - x[:, 2]) / (hi[2] - lo[2])
    D = 0.006 * torch.randn(n, 3, 3, generator=g, device=DEV)
    D[:, 0, 0] -= 0.015 * depth
    D[:, 1, 1] -= 0.015 * depth
    D[:, 2, 2] -= 0.025 * depth
    F = torch.eye(3, device=DEV) + D
    vol = float(torch.prod(hi - lo)) / n
    p = {"x0": x, "u": u, "v": v, "C": C, "F": F, "vol": torch.full((n,), vol, device=DEV),
         "yield": torch.full((n,), YIELD, device=DEV)}
    p["mass"] = mat["rho"] * p["vol"]
    F64, tau, _ = _return_map(F.double(), mat, p["yield"].double())
    p["F"], p["stress"] = F64.float(), tau.float()
    return p


def _load(engine, p):
    for field, name in ((A.FIELD_X_INITIAL, "x0"), (A.FIELD_U, "u"), (A.FIELD_V, "v"), (A.FIELD_C, "C"),
                        (A.FIELD_F, "F"), (A.FIELD_STRESS, "stress"), (A.FIELD_VOL, "vol"), (A.FIELD_MASS, "mass"),
                        (A.FIELD_YIELD, "yield")):
        engine.load(field, p[name])


def _simulator(case, p, mat):
    sim = MPM_Simulator_WARP(case["n"], n_grid=case["grid"], device=DEV)
    sim.set_parameters(material=mat["material"], E=mat["E"], nu=NU, friction_angle=PHI, gravity=GRAVITY,
                       hardening=1, xi=mat["xi"], yield_stress=YIELD)
    _load(sim.engine, p)
    sim.add_surface_collider((0.0, 0.0, _floor(case["grid"])), (0.0, 0.0, 1.0), "sticky", 0.0)
    sim.add_bounding_box()
    return sim


def _scenes(case):
    """The scenes' descriptions (sizes and materials) go with the case, their particles with the seed."""
    return batch_64(seed=7, n_scenes=case["scenes"])


def _scene_material(sc):
    return {"material": sc.material, "mu": sc.mu, "lam": sc.lam, "alpha": _alpha(sc.friction_angle), "xi": sc.xi,
            "rho": sc.density, "dt": sc.dt, "E": sc.E, "hardening": sc.hardening}


def _scene_particles(sc, g):
    p = _particles(sc.n_particles, sc.n_grid, _scene_material(sc), g, (sc.box_lo, sc.box_hi))
    p["yield"] = torch.full((sc.n_particles,), sc.yield_stress, device=DEV)
    return p


def _target(p):
    """Target positions of the gradient case: the column sheared and pushed down."""
    t = p["x0"].double() + p["u"].double()
    t[:, 0] = t[:, 0] + 0.02 * t[:, 2]
    t[:, 2] = 0.98 * t[:, 2]
    return t


def _strains(rows, g):
    """Network inputs as the training set has them, and stress-like targets."""
    B = torch.randn(rows, 3, 3, generator=g, device=DEV)
    B = B + B.transpose(1, 2)
    B = B / B.flatten(1).norm(dim=1)[:, None, None]
    rest = 2.0 * torch.rand(rows, 3, generator=g, device=DEV) - 1.0
    x = torch.cat([B.reshape(rows, 9), rest * torch.tensor([1.4, 0.5, 1.0], device=DEV)], 1)
    iu = torch.tensor([0, 1, 2, 4, 5, 8], device=DEV)
    tr = (B[:, 0, 0] + B[:, 1, 1] + B[:, 2, 2])[:, None]
    y = B.reshape(rows, 9)[:, iu] + 0.7 * tr * torch.tensor([1.0, 0, 0, 1.0, 0, 1.0], device=DEV)
    return x.contiguous(), (y * (1.0 + 0.2 * rest[:, :1])).contiguous()


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind in ("train", "network"):
        x, y = _strains(case["rows"], g)
        return {"kind": kind, "net": StressMLP(DEV, seed=seed % 1000), "x": x, "y": y}
    if kind == "batch":
        scenes = _scenes(case)
        b = BatchedMPM(scenes, device=DEV, chunk_size=128)
        ps = [_scene_particles(sc, g) for sc in scenes]
        _load(b.engine, {k: torch.cat([p[k] for p in ps]) for k in ps[0]})
        return {"kind": kind, "batch": b, "snap": b.engine.snapshot(), "steps": case["steps"], "dt": scenes[0].dt}
    mat = _material(case)
    p = _particles(case["n"], case["grid"], mat, g)
    if kind == "grad":
        lo, hi = _box(case["grid"])
        sc = Scene("rollout", case["n"], case["grid"], 1.0, lo, hi, "sand", mat["E"], NU, PHI, mat["rho"], GRAVITY,
                   1e-4, case["steps"], floor_z=lo[2])
        arrays = tuple(p[k].cpu().numpy() for k in ("x0", "v", "vol", "mass"))
        sand = SandRollout(sc, checkpoint_every=case["every"], device=DEV, particles=arrays,
                           initial={A.FIELD_U: p["u"], A.FIELD_C: p["C"], A.FIELD_F: p["F"],
                                    A.FIELD_STRESS: p["stress"]})
        return {"kind": kind, "sand": sand, "v": p["v"], "target": _target(p), "E": mat["E"]}
    sim = _simulator(case, p, mat)
    st = {"kind": kind, "sim": sim, "dt": mat["dt"], "steps": case.get("steps", 1)}
    if kind == "loop":
        st["frames"] = [((1.0 + 0.1 * k) * p["u"], (1.0 - 0.1 * k) * p["v"], (1.0 - 0.05 * k) * p["stress"])
                        for k in range(case["steps"])]
    if kind == "reduced":
        sim._density = torch.full((case["n"],), mat["rho"], device=DEV)
        sim.load_uvF_from_tensor(p["u"], p["v"], p["F"] - torch.eye(3, device=DEV))
        pick = torch.randperm(case["n"], generator=g, device=DEV)[:case["samples"]].to(torch.int32)
        sim.load_sample_particle_index_from_tensor(pick)
    if kind == "decoder":
        st["label"] = torch.randn(case["label"], generator=g, device=DEV)
        st["decoder"] = _decoder(case, seed)
    st["snap"] = sim.engine.snapshot()
    if kind == "graph":
        for k in range(2):
            sim.p2g2p(k, mat["dt"])
        st["graph"] = sim.engine.graph(case["steps"] - 2, 0.0, mat["dt"])
    return st


def _decoder(case, seed):
    lo, hi = _box(case["grid"])
    a, b = tuple((l + h) / 2 for l, h in zip(lo, hi)), tuple((h - l) / 3 for l, h in zip(lo, hi))
    stats = (lo, hi) if case["siren"] else (a, b)
    return StressDecoder.random(label_dim=case["label"], scale_mlp=case["scale"], siren=case["siren"],
                                seed=seed % 100000, x_stats=stats,
                                q_stats=((-3e3, 10.0, -20.0, -3e3, 5.0, -4e3), (2e3, 500.0, 500.0, 2e3, 500.0, 3e3)),
                                device=DEV)


# --------------------------------------------------------------------------- one pass
def run(st):
    kind = st["kind"]
    if kind == "network":
        return st["net"].forward(st["x"])
    if kind == "train":
        net = st["net"]
        loss = net.train_step(st["x"], st["y"])
        return {"loss": loss, "grad": net.grad, "master": net.master}
    if kind == "grad":
        v0 = st["v"].clone().requires_grad_()
        E = torch.tensor(st["E"], requires_grad=True)
        phi = torch.tensor(PHI, requires_grad=True)
        x = rollout(v0, E, phi, st["sand"])
        ((x - st["target"]) ** 2).sum(1).mean().backward()
        return {"x": x.detach().float(), "v0": v0.grad, "E": E.grad, "phi": phi.grad}
    if kind == "batch":
        b = st["batch"]
        b.engine.restore(st["snap"])
        b.time = 0.0
        for _ in range(st["steps"]):
            b.step(st["dt"])
        return b.engine.export_uvFstress()
    sim = st["sim"]
    if kind == "reduced":
        sim.p2g2p_reduced(0, st["dt"])
        s = sim.mpm_state
        return {"m": s.grid_m, "vin": s.grid_v_in, "vout": s.grid_v_out, "cells": s.neighboring_cells}
    if kind == "decoder":
        sim.load_stress_from_decoder(st["decoder"], st["label"])
        return sim.mpm_state.particle_stress
    sim.engine.restore(st["snap"])
    sim.time = 0.0
    if kind == "loop":
        out = []
        for k, (u, v, stress) in enumerate(st["frames"]):
            sim.load_uvstress_from_tensor(u, v, stress)
            sim.p2g2p(k, st["dt"])
            out.append(sim.export_uvFstress_from_warp())
        return out
    if kind == "graph":
        for k in range(2):
            sim.p2g2p(k, st["dt"])
        st["graph"].replay()
    else:
        for k in range(st["steps"]):
            sim.p2g2p(k, st["dt"])
    return sim.export_uvFstress_from_warp()


# --------------------------------------------------------------------------- bytes and operations
def work(case):
    kind = case["kind"]
    if kind in ("train", "network"):
        rows = case["rows"]
        flops = 2.0 * rows * (12 * 128 + 2 * 128 * 128 + 128 * 6)
        if kind == "network":
            return {"bytes": rows * (12 + 6) * 4.0, "flops": flops}
        # the saved pre-activations need not leave the chip: inputs, targets, parameters and Adam state
        return {"bytes": rows * (12 + 6) * 4.0 + 37264 * 4.0 * 7, "flops": 3.0 * flops}
    if kind == "batch":
        n, steps, per = sum(s.n_particles for s in _scenes(case)), case["steps"], 284.0
    else:
        n, steps, per = case["n"], case.get("steps", 1), 284.0
    if kind == "decoder":
        h, n_in = 3 * case["scale"], case["label"] + 4
        return {"bytes": n * (12 + 4 + 36.0), "flops": 2.0 * n * (n_in * h + 4 * h * h + 6 * h)}
    if kind == "reduced":
        # positions of all, then mass, v and F_disp of the marked (nearly all at these sample counts); grids once
        return {"bytes": n * (24.0 + 4 + 12 + 36 + 36 + 4) + case["grid"] ** 3 * 32.0, "flops": 900.0 * n}
    if kind == "grad":
        # forward state once a substep; backward: the state and the adjoint (33 words) read and written
        return {"bytes": n * steps * (284.0 + 152 + 2 * 132), "flops": 5000.0 * n * steps}
    if case.get("material") == "metal":
        per = 288.0
    io = 60.0 + 96.0 if kind == "loop" else 0.0
    return {"bytes": n * (steps * (per + io) + (0.0 if kind == "loop" else 96.0)), "flops": 1100.0 * n * steps}


# --------------------------------------------------------------------------- float64
def _eig(b):
    """Eigenvalues (n,3) and eigenvectors (n,3,3) of symmetric matrices by Jacobi rotations."""
    a = [[b[:, i, j] for j in range(3)] for i in range(3)]
    one, zero = torch.ones_like(a[0][0]), torch.zeros_like(a[0][0])
    Q = [[one if i == j else zero for j in range(3)] for i in range(3)]
    for _ in range(5):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            th = 0.5 * torch.atan2(2.0 * a[p][q], a[p][p] - a[q][q])
            th = torch.where(th > math.pi / 4, th - math.pi / 2, torch.where(th < -math.pi / 4, th + math.pi / 2, th))
            c, s = torch.cos(th), torch.sin(th)
            for k in range(3):  # columns
                a[k][p], a[k][q] = c * a[k][p] + s * a[k][q], -s * a[k][p] + c * a[k][q]
                Q[k][p], Q[k][q] = c * Q[k][p] + s * Q[k][q], -s * Q[k][p] + c * Q[k][q]
            for k in range(3):  # rows
                a[p][k], a[q][k] = c * a[p][k] + s * a[q][k], -s * a[p][k] + c * a[q][k]
    return (torch.stack([a[i][i] for i in range(3)], 1),
            torch.stack([torch.stack([Q[i][j] for j in range(3)], 1) for i in range(3)], 1))


def _spectral(Q, f):
    return (Q * f[:, None, :]) @ Q.transpose(1, 2)


def _return_map(F, m, yld):
    """(F, Kirchhoff stress, yield stress) after the return map of F."""
    lam_, Q = _eig(F @ F.transpose(1, 2))
    mu, lam = m["mu"], m["lam"]
    if m["material"] == "jelly":
        J = torch.det(F)
        tau = _spectral(Q, 2.0 * mu * (lam_ - lam_.sqrt()))
        return F, tau + (lam * J * (J - 1.0))[:, None, None] * torch.eye(3, dtype=F.dtype, device=F.device), yld
    e = 0.5 * torch.log(lam_)
    tr = e.sum(1, keepdim=True)
    h = e - tr / 3.0
    hn = (h * h).sum(1, keepdim=True).sqrt()
    if m["material"] == "sand":
        dg = hn + (3.0 * lam + 2.0 * mu) / (2.0 * mu) * tr * m["alpha"]
        cone = e - h * (dg / hn.clamp_min(1e-300))
        en = torch.where(dg <= 0.0, e, torch.where(tr > 0.0, torch.zeros_like(e), cone))
        Fn = _spectral(Q, torch.exp(en - e)) @ F
        return Fn, _spectral(Q, 2.0 * mu * en + lam * en.sum(1, keepdim=True)), yld
    y = yld[:, None]
    plastic = 2.0 * mu * hn > y
    dg = hn + 1e-6 - y / (2.0 * mu)
    en = torch.where(plastic, e - h * (dg / (hn + 1e-6)), e)
    Fn = _spectral(Q, torch.exp(en - e)) @ F
    R = _spectral(Q, torch.exp(-e)) @ F
    tau = _spectral(Q, 2.0 * mu * en + lam * en.sum(1, keepdim=True)) @ R
    if m.get("hardening", 1):
        yld = torch.where(plastic[:, 0], yld + 2.0 * mu * m["xi"] * dg[:, 0], yld)
    return Fn, tau, yld


def _stencil(x, grid):
    """base cell, fx and the weights and their derivatives per axis: (n,3), (n,3), (n,3 axes,3 nodes)."""
    gp = x * grid
    base = (gp.detach() - 0.5).to(torch.int64)
    fx = gp - base
    w = torch.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1.0) ** 2, 0.5 * (fx - 0.5) ** 2], 2)
    dw = torch.stack([fx - 1.5, -2.0 * (fx - 1.0), fx - 0.5], 2)
    return base, fx, w, dw


def _nodes(base, fx, w, dw, grid):
    """(flat node index, weight, weight gradient, offset) of the 27 nodes."""
    for i in range(3):
        for j in range(3):
            for k in range(3):
                idx = ((base[:, 0] + i) * grid + base[:, 1] + j) * grid + base[:, 2] + k
                a, b, c = w[:, 0, i], w[:, 1, j], w[:, 2, k]
                g = torch.stack([dw[:, 0, i] * b * c, a * dw[:, 1, j] * c, a * b * dw[:, 2, k]], 1) * grid
                off = torch.stack([i - fx[:, 0], j - fx[:, 1], k - fx[:, 2]], 1) / grid
                yield idx, a * b * c, g, off


def _collide(v, grid, floor):
    """The sticky floor, then the slip walls, on (grid^3, 3) velocities."""
    r = torch.arange(grid, device=v.device)
    ix, iy, iz = (t.reshape(-1) for t in torch.meshgrid(r, r, r, indexing="ij"))
    below = (iz.float() * (1.0 / grid) - torch.tensor(floor, device=v.device)) < 0.0
    v = torch.where(below[:, None], torch.zeros_like(v), v)
    cols = []
    for d, id_ in enumerate((ix, iy, iz)):
        c = v[:, d]
        c = torch.where((id_ < 3) & (c < 0), torch.zeros_like(c), c)
        cols.append(torch.where((id_ >= grid - 3) & (c > 0), torch.zeros_like(c), c))
    return torch.stack(cols, 1)


def _substep(s, m, grid, floor, dt):
    """One explicit substep of a dict of float64 arrays x0, u, v, C, F, stress, vol, mass, yield."""
    x = s["x0"] + s["u"]
    st = _stencil(x, grid)
    mv = s["mass"][:, None]
    acc = torch.zeros(grid ** 3, 4, dtype=x.dtype, device=x.device)
    for idx, w, g, off in _nodes(*st, grid):
        mom = w[:, None] * mv * (s["v"] + (s["C"] @ off[:, :, None])[:, :, 0])
        mom = mom - dt * s["vol"][:, None] * (s["stress"] @ g[:, :, None])[:, :, 0]
        acc = acc.index_add(0, idx, torch.cat([mom, w[:, None] * mv], 1))
    mass = acc[:, 3:]
    live = mass > 1e-15
    gv = torch.where(live, acc[:, :3] / torch.where(live, mass, torch.ones_like(mass)) +
                     dt * torch.tensor(GRAVITY, dtype=x.dtype, device=x.device), torch.zeros_like(acc[:, :3]))
    gv = _collide(gv, grid, floor)
    v, C, G = torch.zeros_like(s["v"]), torch.zeros_like(s["C"]), torch.zeros_like(s["C"])
    for idx, w, g, off in _nodes(*st, grid):
        vn = gv[idx]
        v = v + w[:, None] * vn
        C = C + 4.0 * grid * grid * w[:, None, None] * vn[:, :, None] * off[:, None, :]
        G = G + vn[:, :, None] * g[:, None, :]
    F, tau, yld = _return_map(s["F"] + dt * G @ s["F"], m, s["yield"])
    return {**s, "u": s["u"] + dt * v, "v": v, "C": C, "F": F, "stress": tau, "yield": yld}


def _export(s):
    return s["u"], s["v"], s["F"] - torch.eye(3, dtype=s["F"].dtype, device=s["F"].device), s["stress"]


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind in ("train", "network"):
        return _exact_network(case, seed, g)
    if kind == "batch":
        outs = []
        for sc in _scenes(case):
            s = {k: t.double() for k, t in _scene_particles(sc, g).items()}
            for _ in range(case["steps"]):
                s = _substep(s, _scene_material(sc), sc.n_grid, sc.floor_z, sc.dt)
            outs.append(_export(s))
        return tuple(torch.cat([o[k] for o in outs]).reshape(-1) for k in range(4))
    mat = _material(case)
    grid, floor = case["grid"], _floor(case["grid"])
    p = _particles(case["n"], grid, mat, g)
    s = {k: t.double() for k, t in p.items()}
    if kind == "decoder":
        label = torch.randn(case["label"], generator=g, device=DEV)
        return _exact_decoder(_decoder(case, seed), p["x0"].double(), label.double())
    if kind == "reduced":
        return _exact_reduced(case, s, p, mat, torch.randperm(case["n"], generator=g, device=DEV)[:case["samples"]])
    if kind == "grad":
        return _exact_grad(case, s, p, mat, floor)
    if kind == "loop":
        out = []
        for k in range(case["steps"]):
            s.update(u=((1.0 + 0.1 * k) * p["u"]).double(), v=((1.0 - 0.1 * k) * p["v"]).double(),
                     stress=((1.0 - 0.05 * k) * p["stress"]).double())
            s = _substep(s, mat, grid, floor, mat["dt"])
            out.append(_export(s))
        return out
    for _ in range(case["steps"]):
        s = _substep(s, mat, grid, floor, mat["dt"])
    return _export(s)


def _exact_grad(case, s, p, mat, floor):
    v0 = s["v"].clone().requires_grad_()
    E = torch.tensor(mat["E"], dtype=torch.float64, device=DEV, requires_grad=True)
    phi = torch.tensor(PHI, dtype=torch.float64, device=DEV, requires_grad=True)
    mu, lam = _lame(E)
    sn = torch.sin(phi / 180.0 * 3.14159265)
    m = {**mat, "mu": mu, "lam": lam, "alpha": math.sqrt(2.0 / 3.0) * 2.0 * sn / (3.0 - sn)}
    s = {**s, "v": v0}
    for _ in range(case["steps"]):
        keys = list(s)

        def step(*t):
            o = _substep(dict(zip(keys, t[:len(keys)])), {**m, "mu": t[-3], "lam": t[-2], "alpha": t[-1]}, case["grid"],
                         floor, 1e-4)
            return tuple(o[k] for k in keys)

        o = checkpoint(step, *(s[k] for k in keys), m["mu"], m["lam"], m["alpha"],
                       use_reentrant=False)
        s = dict(zip(keys, o))
    x = s["x0"] + s["u"]
    ((x - _target(p)) ** 2).sum(1).mean().backward()
    return {"x": x.detach(), "v0": v0.grad, "E": E.grad, "phi": phi.grad}


def _exact_reduced(case, s, p, mat, pick):
    grid, dt, floor = case["grid"], mat["dt"], _floor(case["grid"])
    F = (p["F"] - torch.eye(3, device=DEV)).double() + torch.eye(3, dtype=torch.float64, device=DEV)
    x = s["x0"] + s["u"]
    base32 = ((p["x0"] + p["u"]) * float(grid) - 0.5).to(torch.int64)
    marks = torch.zeros(grid, grid, grid, dtype=torch.int32, device=DEV)
    r = torch.arange(-2, 3, device=DEV)
    for i in r:
        for j in r:
            for k in r:
                c = base32[pick] + torch.stack([i, j, k])
                c = c[((c >= 0) & (c < grid)).all(1)]
                marks[c[:, 0], c[:, 1], c[:, 2]] = 1
    on = marks[base32[:, 0], base32[:, 1], base32[:, 2]] > 0
    lam_, Q = _eig(F @ F.transpose(1, 2))
    mu, lam = mat["mu"], mat["lam"]
    if mat["material"] == "sand":
        e = 0.5 * torch.log(lam_)
        tau = _spectral(Q, 2.0 * mu * e + lam * e.sum(1, keepdim=True))
    else:
        J = torch.det(F)
        tau = _spectral(Q, 2.0 * mu * (lam_ - lam_.sqrt())) + \
            (lam * J * (J - 1.0))[:, None, None] * torch.eye(3, dtype=torch.float64, device=DEV)
    acc = torch.zeros(grid ** 3, 4, dtype=torch.float64, device=DEV)
    mass, vol = s["mass"] * on, s["mass"] / mat["rho"] * on
    st = _stencil(x, grid)
    for idx, w, g, _ in _nodes(*st, grid):
        mom = (w * mass)[:, None] * s["v"] - dt * vol[:, None] * (tau @ g[:, :, None])[:, :, 0]
        acc.index_add_(0, idx, torch.cat([mom, (w * mass)[:, None]], 1))
    m = acc[:, 3:]
    live = (m > 1e-10) & (marks.reshape(-1, 1) > 0)
    gv = torch.where(live, acc[:, :3] / torch.where(live, m, torch.ones_like(m)) +
                     dt * torch.tensor(GRAVITY, dtype=torch.float64, device=DEV), torch.zeros_like(acc[:, :3]))
    gv = _collide(gv, grid, floor)
    shape = (grid, grid, grid)
    return {"m": m.reshape(shape), "vin": acc[:, :3].reshape(*shape, 3), "vout": gv.reshape(*shape, 3), "cells": marks}


def _exact_decoder(dec, x, label):
    sd = {k: v.double().to(DEV) for k, v in dec.state_dict.items()}
    if dec.siren:
        lo, hi = sd["prepare.min_x_torch"], sd["prepare.max_x_torch"]
        x = 2.0 * (x - lo) / (hi - lo) - 1.0
    else:
        x = (x - sd["prepare.mean_x_torch"]) / sd["prepare.std_x_torch"]
    h = torch.cat([label.expand(x.shape[0], -1), x, torch.full_like(x[:, :1], PHI)], 1)
    for name in ("dec0", "dec1", "dec2", "dec3", "dec4"):
        h = h @ sd[name + ".weight"].T + sd[name + ".bias"]
        h = torch.sin(dec.omega_0 * h) if dec.siren else torch.nn.functional.elu(h)
    q = h @ sd["enc.weight"].T + sd["enc.bias"]
    q = sd["invStandardizeQ.mean_q_torch"] + q * sd["invStandardizeQ.std_q_torch"]
    return q[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(-1, 3, 3)


def _exact_network(case, seed, g):
    x, y = _strains(case["rows"], g)
    net = StressMLP(DEV, seed=seed % 1000)  # the initial parameters only
    # the weights as the network holds them (bf16), the arithmetic in 64 bits
    m = net.master.double()
    flat = torch.cat([net.master[:W_COUNT].bfloat16().double(), m[W_COUNT:]]).requires_grad_()
    shapes, parts, o = [(128, 16), (128, 128), (128, 128), (16, 128), (128,), (128,), (128,), (16,)], [], 0
    for shape in shapes:
        size = math.prod(shape)
        parts.append(flat[o:o + size].reshape(shape))
        o += size
    h = torch.nn.functional.pad(x.double(), (0, 4))
    for layer in range(4):
        h = h @ parts[layer].T + parts[4 + layer]
        if layer < 3:
            h = torch.nn.functional.silu(h)
    out = h[:, :6]
    if case["kind"] == "network":
        return out.detach()
    loss = ((out - y.double()) ** 2).mean()
    loss.backward()
    return {"loss": loss.detach().reshape(1), "grad": flat.grad, "master": None}
