"""The sort's prefix over sums of sums, on grids of more than 2^20 buckets (grid blocks):
particles over the whole grid, the groups' first and last blocks included.  Grid mass
against a float64 scatter over two substeps, and every particle in some cell."""
import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S

from helpers import gpu_sim, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_grid", [404, 408, 412])  # 101^3 < 2^20 < 102^3, 103^3 buckets
def test_sort_over_sums_of_sums(cuda, n_grid):
    rng = np.random.default_rng(n_grid)
    n = 4000
    sc = S.small_column(n, n_grid, gravity=(0.0, 0.0, 0.0))
    nb = (n_grid + 3) // 4
    cell = rng.integers(0, n_grid - 2, (n, 3))
    # blocks on both sides of the edges between groups of 256 x 512 buckets
    edges = np.arange(1, nb ** 3 // 131072 + 1) * 131072
    blk = np.unique(np.concatenate([edges - 1, edges, edges + 1, [0, 1, nb ** 3 - 1]]))
    blk = blk[blk < nb ** 3]
    at = np.stack([blk // (nb * nb), blk // nb % nb, blk % nb], 1) * 4
    cell[:len(blk)] = np.minimum(at, n_grid - 3)
    x0 = ((cell + 0.5 + rng.uniform(0.05, 0.95, (n, 3))) / n_grid).astype(np.float32)
    x0[100::200] += 2.0  # outside the domain
    mass = rng.uniform(1.0, 2.0, n).astype(np.float32)
    sim = gpu_sim(sc, x0=x0, v0=np.zeros((n, 3), np.float32), vol=np.full(n, 1e-9, np.float32), mass=mass,
                  colliders=False)
    sim.on_error = "ignore"
    e = sim.engine
    gp = (x0 * np.float32(n_grid)).astype(np.float64)  # the grid coordinate as the kernels round it
    inside = (x0 < 1.5).all(1)
    base = np.trunc(gp - 0.5).astype(np.int64)
    fx = gp - base
    w = np.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2], -1)
    want = torch.zeros(n_grid ** 3, dtype=torch.float64, device=cuda)
    for q in range(27):
        a, b, c = q // 9, q // 3 % 3, q % 3
        node = ((base[:, 0] + a) * n_grid + base[:, 1] + b) * n_grid + base[:, 2] + c
        wm = w[:, 0, a] * w[:, 1, b] * w[:, 2, c] * mass
        want.index_add_(0, torch.from_numpy(node[inside]).to(cuda), torch.from_numpy(wm[inside]).to(cuda))
    touched = want.nonzero().ravel()
    for _ in range(2):  # at rest and without gravity nothing moves; the second sort has G2P's counts
        e.stage("sort")
        e.stage("p2g", dt=sc.dt)
        gm = e.export_grid(0)[0].ravel()
        assert rel(gm[touched].cpu().numpy(), want[touched].cpu().numpy()) < 1e-5
        assert int((gm != 0).sum()) == touched.numel()
        e.stage("grid", time=0.0, dt=sc.dt)
        e.stage("g2p", dt=sc.dt)
    assert torch.equal(e.export(A.FIELD_MASS).cpu(), torch.from_numpy(mass))
    assert e.status() == A.ST_OUT_OF_DOMAIN
    e.clear_status()
