"""The exports' row layout at warp and CTA edges: every field of a state whose
slots are in another order than the user's, exactly as loaded."""
import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S

from helpers import gpu_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 127, 129, 255, 257, 1000])
def test_exports_return_what_was_loaded(cuda, n):
    rng = np.random.default_rng(n)
    sc = S.small_column(n, 16)
    sim = gpu_sim(sc)
    e = sim.engine
    e.substep_raw(0.0, sc.dt)  # sorts the slots by cell
    loaded = {}
    for f in (A.FIELD_U, A.FIELD_V, A.FIELD_C, A.FIELD_F, A.FIELD_STRESS, A.FIELD_MASS, A.FIELD_VOL, A.FIELD_YIELD):
        loaded[f] = torch.from_numpy(rng.normal(size=n * A.FIELD_COMPONENTS[f]).astype(np.float32)).to(cuda)
        e.load(f, loaded[f])
    for f, t in loaded.items():
        out = torch.full((t.numel() + 64,), 7.0, device=cuda)
        e.export(f, out[:t.numel()])
        assert torch.equal(out[:t.numel()], t), f
        assert bool((out[t.numel():] == 7.0).all()), f  # nothing past the last row
    x0 = torch.from_numpy(sc.particles()[0]).to(cuda).reshape(-1)
    assert torch.equal(e.export(A.FIELD_X), x0 + loaded[A.FIELD_U])
    eye = torch.eye(3, device=cuda).reshape(-1).repeat(n)
    fd = loaded[A.FIELD_F] - eye
    assert torch.equal(e.export(A.FIELD_F_DISP), fd)
    pad = 64
    outs = [torch.full((n * c + pad,), 7.0, device=cuda) for c in (3, 3, 9, 9)]
    e.export_uvFstress(tuple(o[:o.numel() - pad] for o in outs))
    for o, want in zip(outs, (loaded[A.FIELD_U], loaded[A.FIELD_V], fd, loaded[A.FIELD_STRESS])):
        assert torch.equal(o[:want.numel()], want)
        assert bool((o[want.numel():] == 7.0).all())
    e.load_uvstress(loaded[A.FIELD_V], loaded[A.FIELD_U], loaded[A.FIELD_C])
    assert torch.equal(e.export(A.FIELD_U), loaded[A.FIELD_V])
    assert torch.equal(e.export(A.FIELD_STRESS), loaded[A.FIELD_C])
    assert torch.equal(e.export(A.FIELD_C), loaded[A.FIELD_C])
