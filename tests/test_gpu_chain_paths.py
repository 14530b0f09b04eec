"""Kernels that are started behind one another without waiting on the host, on every path
but the ordered substep: what a program gets that queues its calls back to back (and, for
substeps, from a graph) against a process that runs every launch to its end before the
next (CUDA_LAUNCH_BLOCKING=1).  A kernel that did not wait for the one before it would read what
that one is still writing: moved colliders, the state just loaded, parameters after Adam.

Tolerances: sums over float atomics differ by rounding; 1e-5 relative a substep is the
per-substep bar of these kernels (4 substeps here), as for the grids; the gradient's
is derived in test_gpu_adjoint_layout (2.5e-5 over two substeps, four here); Adam's first
steps turn a gradient's sign into a step, so entries below the gradient's rounding may
differ by whole steps: 1 % of the update.  Whatever has no such sums is equal bit for bit."""
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

if __name__ == "__main__":
    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S
from reduced_mpm_stress_training_gb300.adjoint import SandRollout
from reduced_mpm_stress_training_gb300.decoder import StressDecoder
from reduced_mpm_stress_training_gb300.surrogate import StressMLP, StressSurrogate

from helpers import gpu_sim, rel

pytestmark = pytest.mark.gpu

N, GRID, STEPS = 20000, 32, 4
SUBSTEP, GRADIENT, ADAM, BITS = 1e-5 * STEPS, 5e-5, 1e-2, 0.0


def _gen(seed):
    return torch.Generator(device="cuda:0").manual_seed(seed)


def _sim(material="sand"):
    sc = S.small_column(N, GRID, seed=3, floor_z=0.15, v0_sigma=0.1, material=material)
    sim = gpu_sim(sc)
    sim.set_parameters(density=sc.density)
    # moves between substeps, on the device
    sim.set_velocity_on_infinite_plane((0.0, 0.0, 0.4), (0.0, 0.0, 1.0), (0.5, 0.0, 0.0), 0.05)
    F = torch.eye(3, device="cuda:0") + 0.02 * torch.randn(N, 3, 3, generator=_gen(1), device="cuda:0")
    sim.load_F_from_tensor(F)
    return sim, sc


def _state(e, tol, out, name, fields=("X", "V", "F")):
    for f in fields:
        out[f"{name}.{f}"] = (e.export(getattr(A, "FIELD_" + f)).cpu().numpy(), tol)


def substeps(out):
    for material in ("sand", "metal", "jelly"):
        sim, sc = _sim(material)
        for k in range(STEPS):
            sim.p2g2p(k, sc.dt)
            sim.engine.export(A.FIELD_STRESS)
        _state(sim.engine, SUBSTEP, out, material)


def graph(out):
    sim, sc = _sim()
    sim.p2g2p(0, sc.dt)
    g = sim.engine.graph(2, 0.0, sc.dt)
    g.replay()
    sim.p2g2p(3, sc.dt)
    _state(sim.engine, SUBSTEP, out, "graph")


def surrogate(out):
    sim, sc = _sim()
    sim.engine.set_stress_surrogate(StressSurrogate(StressMLP("cuda:0", seed=1), tol=0.0))
    for k in range(STEPS):
        sim.p2g2p(k, sc.dt)
    _state(sim.engine, SUBSTEP, out, "surrogate")


def learned_loop(out):
    sim, sc = _sim("jelly")
    dec = StressDecoder.random(label_dim=4, seed=3, device="cuda:0")
    for k in range(STEPS):
        sim.load_uvstress_from_tensor(*(0.01 * torch.randn(N, c, generator=_gen(10 * k + c), device="cuda:0")
                                        for c in (3, 3, 9)))
        sim.load_stress_from_decoder(dec, torch.randn(4, generator=_gen(k), device="cuda:0"))
        out[f"loop.decoded{k}"] = (sim.engine.export(A.FIELD_STRESS).cpu().numpy(), BITS)
        sim.p2g2p(k, sc.dt)
        u, v, F, stress = sim.export_uvFstress_from_warp()
        out[f"loop.v{k}"] = (v.cpu().numpy(), SUBSTEP)
    out["loop.frame"] = (sim.export_frame_arrays()["v"], SUBSTEP)


def reduced(out):
    sim, sc = _sim()
    sim.p2g2p(0, sc.dt)
    sim.load_sample_particle_index_from_tensor(torch.arange(0, N, 50, dtype=torch.int32))
    for k in range(2):
        fd = 0.02 * torch.randn(N, 3, 3, generator=_gen(k), device="cuda:0")
        u = 0.01 * torch.randn(N, 3, generator=_gen(20 + k), device="cuda:0")
        sim.load_uvF_from_tensor(u, torch.randn(N, 3, generator=_gen(30 + k), device="cuda:0"), fd)
        sim.p2g2p_reduced(k, sc.dt)
        sim.experiment_for_C()
        s = sim.mpm_state
        for g in ("grid_m", "grid_v_in", "grid_v_out"):
            out[f"reduced.{g}{k}"] = (getattr(s, g).cpu().numpy(), 1e-5)
        for g in ("neighboring_cells", "neighboring_cells_grid_v"):
            out[f"reduced.{g}{k}"] = (getattr(s, g).cpu().numpy(), BITS)
        sim.g2p_sample(sc.dt)
        _state(sim.engine, 1e-5, out, f"reduced.sampled{k}")


def gradient(out):
    for tape in (True, False):
        sc = S.small_column(3000, GRID, seed=5, floor_z=0.15, v0_sigma=0.1)
        sc.substeps = 4
        sand = SandRollout(sc, checkpoint_every=2, device="cuda:0", grid_tape=tape)
        sand.forward(sand.v0_default, sc.E, sc.friction_angle)
        sand.backward(torch.randn(3000, A.ADJ_WORDS, generator=_gen(4), device="cuda:0"))
        out[f"gradient{int(tape)}"] = (sand.state_bar[:, :33].cpu().numpy(), GRADIENT)


def training(out):
    for tc in (True, False):
        net = StressMLP("cuda:0", seed=2, tensor_memory=tc)
        first = net.master.clone()
        for k in range(STEPS):
            x = torch.randn(3001, 12, generator=_gen(40 + k), device="cuda:0")
            y = torch.randn(3001, 6, generator=_gen(50 + k), device="cuda:0")
            net.train_step(x, y)
        net.check_tensor_cores()
        out[f"training{int(tc)}.update"] = ((net.master - first).cpu().numpy(), ADAM)
        held = StressMLP("cuda:0", seed=9, tensor_memory=tc)
        ys = [held.forward(torch.randn(999, 12, generator=_gen(60 + k), device="cuda:0")) for k in range(STEPS)]
        out[f"training{int(tc)}.forward"] = (torch.stack(ys).cpu().numpy(), BITS)


PATHS = (substeps, graph, surrogate, learned_loop, reduced, gradient, training)


@pytest.fixture(scope="module")
def one_at_a_time(cuda, tmp_path_factory):
    path = str(tmp_path_factory.mktemp("chain") / "out.npz")
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1")
    r = subprocess.run([sys.executable, os.path.abspath(__file__), path], env=env, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(path)


@pytest.mark.parametrize("run", PATHS, ids=lambda f: f.__name__)
def test_calls_queued_back_to_back(cuda, one_at_a_time, run):
    out = {}
    run(out)
    for name, (got, tol) in out.items():
        want = one_at_a_time[name]
        assert np.isfinite(want).all() and want.any(), name
        if tol == BITS:
            assert np.array_equal(got, want), name
        else:
            assert rel(got, want) <= tol, (name, rel(got, want))


if __name__ == "__main__":
    results = {}
    for path in PATHS:
        path(results)
    np.savez(sys.argv[1], **{name: value for name, (value, _) in results.items()})
