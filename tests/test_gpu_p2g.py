"""P2G and G2P at the edges of their work split.  P2G against the float32 oracle: particle
counts around a warp's batch of 32 and its three groups, in one cell, in one
x-slab of a grid block, in one block and over blocks that the grid cuts off;
and blocks whose slabs are empty.

Tolerance: the per-substep bar of the parity tests, 1e-5 relative L2 on grid
mass and momentum (a node sums at most a few hundred rounded terms, about
1e-6 of their norm in float32).
"""
import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S

from helpers import gpu_sim, gpu_state, oracle_sim, rel

pytestmark = pytest.mark.gpu

N_GRID = 18  # the last 4x4x4 block of an axis holds two node planes
TOL = 1e-5


def _cells(where, n, rng):
    """Base cells (n, 3): block (1, 2, 1) spans cells 4-7, 8-11, 4-7."""
    lo, hi = {"cell": ((6, 9, 5), (7, 10, 6)), "slab": ((5, 8, 4), (6, 12, 8)), "block": ((4, 8, 4), (8, 12, 8)),
              "two_slabs": ((4, 8, 4), (8, 12, 8)), "edge": ((13, 13, 13), (16, 16, 16))}[where]
    c = np.stack([rng.integers(lo[d], hi[d], n) for d in range(3)], 1)
    if where == "two_slabs":  # slabs 1 and 2 stay empty
        c[:, 0] = np.where(c[:, 0] < 6, 4, 7)
    return c


@pytest.mark.parametrize("where", ["cell", "slab", "block", "two_slabs", "edge"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 31, 32, 33, 63, 64, 65, 97, 300])
def test_p2g_split_matches_oracle(cuda, where, n):
    rng = np.random.default_rng(1000 + n)
    sc = S.small_column(n, N_GRID)
    # x / dx = base + 0.5 + [0.01, 0.99): clear of the cell borders
    x0 = ((_cells(where, n, rng) + 0.5 + rng.uniform(0.01, 0.99, (n, 3))) / N_GRID).astype(np.float32)
    v = rng.normal(size=(n, 3)).astype(np.float32)
    Cm = (0.5 * rng.normal(size=(n, 9))).astype(np.float32)
    tau = (1e3 * rng.normal(size=(n, 9))).astype(np.float32)
    vol = np.full(n, 1e-5, np.float32)
    mass = (rng.uniform(1.0, 2.0, n) * 1e-2).astype(np.float32)
    sim = gpu_sim(sc, x0=x0, v0=v, vol=vol, mass=mass)
    sim.load_C_from_tensor(torch.from_numpy(Cm))
    sim.load_uvstress_from_tensor(torch.zeros(n, 3), torch.from_numpy(v), torch.from_numpy(tau))
    ref = oracle_sim(sc, x0=x0, v0=v, vol=vol, mass=mass)
    ref.C[:] = Cm
    ref.stress[:] = tau
    e = sim.engine
    for _ in range(2):  # the second time the previous grid has to be cleared
        e.stage("sort")
        e.stage("p2g", dt=sc.dt)
        gm, gvin, _ = e.export_grid(0)
        e.buf.keys_valid = 0
        ref.stage_p2g(sc.dt)
        assert rel(gm.cpu().numpy(), ref.grid_m) < TOL
        assert rel(gvin.cpu().numpy(), ref.grid_v_in) < TOL
        e.stage("grid", time=0.0, dt=sc.dt)
    assert e.status() == 0


@pytest.mark.parametrize("material", ["sand", "metal", "jelly"])
@pytest.mark.parametrize("chunk", [32, 64, 128, 256])
def test_substep_matches_its_stages(cuda, chunk, material):
    """mpm_p2g2p's own G2P form against the mpm_g2p stage over three substeps, at
    chunks that end inside a warp, blocks that the grid cuts off, particles that
    change cell and block, and one outside the domain.  1e-5 relative, the
    per-substep bar (the two round differently)."""
    rng = np.random.default_rng(chunk)
    n = 2 * chunk + 37
    kw = dict(E=2e5, density=2000.0, yield_stress=2e3, hardening=1, xi=0.1) if material == "metal" else {}
    sc = S.small_column(n, N_GRID, material="metal" if material == "metal" else "sand", **kw)
    sc.material = material
    x0 = (rng.uniform(4.0, 15.4, (n, 3)) / N_GRID).astype(np.float32)
    x0[: chunk + 5] = (rng.uniform(13.6, 15.4, (chunk + 5, 3)) / N_GRID).astype(np.float32)  # one edge block
    x0[-1] = 1.5
    v = (40.0 * rng.normal(size=(n, 3))).astype(np.float32)  # up to about half a cell a substep
    F = (np.eye(3) + 0.02 * rng.normal(size=(n, 3, 3)) - 0.03 * np.eye(3)).astype(np.float32)
    vol = np.full(n, 1e-5, np.float32)
    mass = np.full(n, 2e-2, np.float32)
    out = []
    for whole in (True, False):
        sim = gpu_sim(sc, chunk_size=chunk, x0=x0, v0=v, vol=vol, mass=mass)
        sim.on_error = "ignore"
        sim.load_F_from_tensor(torch.from_numpy(F))
        e = sim.engine
        for _ in range(3):
            if whole:
                e.substep_raw(0.0, sc.dt)
            else:
                for name in ("sort", "p2g", "grid", "g2p"):
                    e.stage(name, time=0.0, dt=sc.dt)
        out.append(gpu_state(sim))
        e.clear_status()
    for f in ("x", "v", "F", "yield_"):
        assert rel(out[0][f], out[1][f]) < TOL, f
    assert np.isfinite(out[0]["stress"]).all()


@pytest.mark.parametrize("n_grid", [4, 15, 16, 80, 84, 200, 204])
def test_sort_over_grid_sizes(cuda, n_grid):
    """The sort's scan at its changes of form (8,192 and 131,072 buckets) and at
    grids of one to a few CTAs: particles over the whole grid, first and last
    blocks included, some outside; two substeps, the second on G2P's counts.
    Grid mass against the oracle, and every particle in some cell."""
    rng = np.random.default_rng(n_grid)
    n = 3000
    sc = S.small_column(n, n_grid, gravity=(0.0, 0.0, 0.0))
    x0 = ((0.5 + rng.uniform(0.01, n_grid - 2.01, (n, 3))) / n_grid).astype(np.float32)
    x0[0] = 0.51 / n_grid
    x0[1] = (n_grid - 1.51) / n_grid
    x0[7::100] += 2.0  # outside the domain
    inside = (x0 < 1.5).all(1)
    vol = np.full(n, 1e-6, np.float32)
    mass = rng.uniform(1.0, 2.0, n).astype(np.float32)
    v = np.zeros((n, 3), np.float32)
    sim = gpu_sim(sc, x0=x0, v0=v, vol=vol, mass=mass, colliders=False)
    sim.on_error = "ignore"
    k = int(inside.sum())
    ref = oracle_sim(S.small_column(k, n_grid, gravity=(0.0, 0.0, 0.0)), x0=x0[inside], v0=v[inside], vol=vol[inside],
                     mass=mass[inside], colliders=False)
    ref.stage_p2g(sc.dt)
    e = sim.engine
    for _ in range(2):  # at rest and without gravity nothing moves
        e.stage("sort")
        e.stage("p2g", dt=sc.dt)
        gm, _, _ = e.export_grid(0)
        assert rel(gm.cpu().numpy(), ref.grid_m) < TOL
        e.stage("grid", time=0.0, dt=sc.dt)
        e.stage("g2p", dt=sc.dt)
    assert torch.equal(e.export(A.FIELD_MASS).cpu(), torch.from_numpy(mass))
    e.clear_status()
