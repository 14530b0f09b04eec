"""The frame export and the u, v, stress load walk the particles in user order and the
record's pair arrays one after another: every row, at the edges of their blocks, for
particles whose user order is no order of the cells."""
import ctypes as C

import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S

from helpers import gpu_sim

pytestmark = pytest.mark.gpu

FIELDS = {A.FIELD_X_INITIAL: 3, A.FIELD_U: 3, A.FIELD_V: 3, A.FIELD_C: 9, A.FIELD_F: 9, A.FIELD_STRESS: 9,
          A.FIELD_MASS: 1, A.FIELD_VOL: 1, A.FIELD_YIELD: 1}


def _moved(n, cuda):
    sc = S.small_column(n, 24, v0_sigma=0.5)
    sim = gpu_sim(sc)
    sim.engine.load(A.FIELD_MASS, torch.rand(n, device=cuda) + 1.0)
    for k in range(2):
        sim.p2g2p(k, sc.dt)
    return sim


def _fields(e, n):
    return {f: e.export(f).cpu().numpy().reshape(n, c) for f, c in FIELDS.items()}


@pytest.mark.parametrize("n", [1, 255, 256, 257, 3000])
def test_frame_rows(cuda, n):
    e = _moved(n, cuda).engine
    out = torch.full((34 * n + 64,), 7.0, device=cuda)
    A.check(e.lib.mpm_export_frame(C.byref(e.buf), out.data_ptr(), e.stream), "mpm_export_frame")
    f = _fields(e, n)
    eye = np.eye(3, dtype=np.float32).reshape(1, 9)
    want = np.concatenate([f[A.FIELD_X_INITIAL], f[A.FIELD_U], f[A.FIELD_MASS], f[A.FIELD_F] - eye,
                           f[A.FIELD_STRESS][:, [0, 1, 2, 4, 5, 8]], f[A.FIELD_V], f[A.FIELD_C]], 1).T
    got = out.cpu().numpy()
    assert np.array_equal(got[:34 * n].reshape(34, n), want)
    assert (got[34 * n:] == 7.0).all()


@pytest.mark.parametrize("n", [1, 255, 256, 257, 3000])
def test_load_writes_its_words_alone(cuda, n):
    e = _moved(n, cuda).engine
    want = _fields(e, n)
    g = torch.Generator(device=cuda).manual_seed(n)
    new = [torch.randn(n, c, generator=g, device=cuda) for c in (3, 3, 9)]
    e.load_uvstress(*new)
    for field, t in zip((A.FIELD_U, A.FIELD_V, A.FIELD_STRESS), new):
        want[field] = t.cpu().numpy()
    got = _fields(e, n)
    for field in FIELDS:
        assert np.array_equal(got[field], want[field]), field
