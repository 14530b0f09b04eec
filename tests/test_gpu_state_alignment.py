"""State buffers that are aligned to 16 bytes and no more: every path that moves records
gives what it gives on aligned buffers; buffers of less alignment are refused."""
import ctypes as C

import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S
from reduced_mpm_stress_training_gb300.decoder import StressDecoder
from reduced_mpm_stress_training_gb300.surrogate import StressMLP, StressSurrogate

from helpers import gpu_sim, gpu_state, rel

pytestmark = pytest.mark.gpu

N, GRID = 3000, 24
TOL = 1e-5  # the per-substep bar: the two buffers run forms that round differently
FIELDS = ("u", "v", "C", "F", "stress", "x", "yield_")


def _sim(offset, cuda, **kw):
    sc = S.small_column(N, GRID, v0_sigma=0.5)
    sim = gpu_sim(sc, **kw)
    sim.set_parameters(density=sc.density)
    e = sim.engine
    if offset is not None:
        fields = {f: e.export(f) for f in (A.FIELD_X_INITIAL, A.FIELD_V, A.FIELD_VOL, A.FIELD_MASS)}
        sim.moved = [torch.zeros(e.plan.state_bytes + 256, dtype=torch.uint8, device=cuda) for _ in range(2)]
        for k, t in enumerate(sim.moved):
            assert t.data_ptr() % 256 == 0
            e.buf.state[k] = t.data_ptr() + offset
        if offset % 16 == 0:
            e.reinit()
            for f, t in fields.items():
                e.load(f, t)
    F = np.eye(3, dtype=np.float32) + 0.02 * np.random.default_rng(1).standard_normal((N, 3, 3)).astype(np.float32)
    if offset is None or offset % 16 == 0:
        sim.load_F_from_tensor(torch.from_numpy(F))
    return sim, sc


def _pair(cuda, **kw):
    return _sim(None, cuda, **kw), _sim(16, cuda, **kw)


def _equal(a, b, fields=FIELDS):
    ga, gb = gpu_state(a), gpu_state(b)
    for f in fields:
        assert np.array_equal(ga[f], gb[f]), f


@pytest.mark.parametrize("chunk", [32, 128])
def test_substeps(cuda, chunk):
    (a, sc), (b, _) = _pair(cuda, chunk_size=chunk)
    for sim in (a, b):
        for k in range(3):
            sim.p2g2p(k, sc.dt)
        sim.check_status()
    ga, gb = gpu_state(a), gpu_state(b)
    for f in ("x", "v", "F", "C"):
        assert rel(ga[f], gb[f]) < TOL, f


def test_ordered_substeps_and_transfers(cuda):
    (a, sc), (b, _) = _pair(cuda)
    out = []
    for sim in (a, b):
        e = sim.engine
        e.ordered = True
        for k in range(3):
            e.substep_raw(0.0, sc.dt)
        frame = torch.zeros(34 * N, device=cuda)
        A.check(e.lib.mpm_export_frame(C.byref(e.buf), frame.data_ptr(), e.stream), "mpm_export_frame")
        out.append([frame, *e.export_uvFstress()])
    _equal(a, b)
    assert all(torch.equal(p, q) for p, q in zip(*out))
    g = torch.Generator(device=cuda).manual_seed(2)
    new = [torch.randn(N, c, generator=g, device=cuda) for c in (3, 3, 9)]
    for sim in (a, b):
        sim.engine.load_uvstress(*new)
    _equal(a, b)


@pytest.mark.parametrize("scale_mlp", [10, 20])  # widths 30 (tensor cores) and 60
def test_decoder_and_reduced_substep(cuda, scale_mlp):
    (a, sc), (b, _) = _pair(cuda)
    dec = StressDecoder.random(label_dim=4, scale_mlp=scale_mlp, seed=3, device=cuda)
    label = torch.randn(4, generator=torch.Generator(device=cuda).manual_seed(3), device=cuda)
    for sim in (a, b):
        sim.load_stress_from_decoder(dec, label)
    _equal(a, b)
    assert gpu_state(b)["stress"].any()
    zero = torch.zeros(N, 3, device=cuda)
    fd = 0.02 * torch.randn(N, 3, 3, generator=torch.Generator(device=cuda).manual_seed(4), device=cuda)
    for sim in (a, b):
        sim.load_uvF_from_tensor(zero, zero, fd)
        sim.load_sample_particle_index_from_tensor(torch.arange(0, N, 40, dtype=torch.int32))
        sim.p2g2p_reduced(0, sc.dt)
        sim.check_status()
    _equal(a, b, ("F", "u", "v"))
    for name in ("grid_m", "grid_v_in", "grid_v_out"):
        assert rel(getattr(b.mpm_state, name).cpu().numpy(), getattr(a.mpm_state, name).cpu().numpy()) < TOL, name


def test_surrogate_substep(cuda):
    (a, sc), (b, _) = _pair(cuda)
    sur = StressSurrogate(StressMLP(cuda, seed=1), tol=0.0)  # an exact gate: every particle takes the return map
    for sim in (a, b):
        sim.engine.set_stress_surrogate(sur)
        for k in range(2):
            sim.p2g2p(k, sc.dt)
        sim.check_status()
    ga, gb = gpu_state(a), gpu_state(b)
    for f in ("x", "v", "F", "C"):
        assert rel(ga[f], gb[f]) < TOL, f


@pytest.mark.parametrize("offset", [4, 8])
def test_less_alignment_is_refused(cuda, offset):
    sim, sc = _sim(offset, cuda)
    e = sim.engine
    b = C.byref(e.buf)
    assert e.lib.mpm_p2g2p(b, 0.0, sc.dt, e.stream) == A.MPM_ERR_ARG
    noalloc = e.lib.mpm_p2g2p_noalloc
    noalloc.argtypes = [C.POINTER(A.MpmBuffers), C.c_float, C.c_float, C.c_void_p]
    assert noalloc(b, 0.0, sc.dt, e.stream) == A.MPM_ERR_ARG
    assert e.lib.mpm_init(b, e.stream) == A.MPM_ERR_ARG
