"""The kernels are launched so that each may start while the one before it still
runs, and wait for it themselves.  A substep graph captured right behind copies
and clears of the state (nodes that are no kernels), and eager substeps between
other work on the stream, give bit for bit what substeps with a synchronisation
after each give (in the ordered mode, whose sums do not vary from run to run)."""
import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S
from reduced_mpm_stress_training_gb300.batched import scene_params
from reduced_mpm_stress_training_gb300.engine import MPMEngine

pytestmark = pytest.mark.gpu

STEPS = 6


def _engine(n, cuda):
    sc = S.small_column(n, 32, seed=3, floor_z=0.15, v0_sigma=0.1)
    e = MPMEngine([scene_params(sc)], device=cuda)
    e.ordered = True
    x0, v0, vol, mass = (torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in sc.particles())
    for field, t in ((A.FIELD_X_INITIAL, x0), (A.FIELD_V, v0), (A.FIELD_VOL, vol), (A.FIELD_MASS, mass)):
        e.load(field, t)
    return e, float(sc.dt)


def _fields(e):
    return [e.export(f).cpu() for f in (A.FIELD_U, A.FIELD_V, A.FIELD_C, A.FIELD_F, A.FIELD_STRESS)]


@pytest.mark.parametrize("n", [1, 129, 20000])
def test_overlapping_launches_change_nothing(cuda, n):
    e, dt = _engine(n, cuda)
    e.substep_raw(0.0, dt)
    snap = e.snapshot()
    for _ in range(STEPS):
        e.substep_raw(0.0, dt)
        torch.cuda.synchronize()
    want = _fields(e)

    e.restore(snap)
    noise = torch.zeros(1 << 20, device=cuda)
    for k in range(STEPS):
        noise += 1.0
        e.substep_raw(0.0, dt)
        e.export(A.FIELD_U)
    eager = _fields(e)

    graph = torch.cuda.CUDAGraph()
    e.restore(snap)
    with torch.cuda.graph(graph):
        e.restore(snap)
        for _ in range(STEPS):
            e.substep_raw(0.0, dt)
    graph.replay()
    replay = _fields(e)
    for got in (eager, replay):
        for a, b in zip(got, want):
            assert torch.equal(a, b)
