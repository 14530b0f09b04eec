"""Stress of the reduced substep over strains of any size: F_disp comes from the caller
(a model's prediction), so singular values far from 1 and far apart are valid inputs.

Each particle has a stencil of its own, so the force that the grid receives shows
each particle's stress error alone.  Bound on the median error relative to float64:
8 units of 2^-24 times s_max / s_min, as an SVD with errors of a few units of s_max gives
(an error that grows with the square of s_max / s_min, or with 1 / s_min^2, is above)."""
import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import MPM_Simulator_WARP
from reduced_mpm_stress_training_gb300 import _capi as A

pytestmark = pytest.mark.gpu

N, M = 64, 12
E, NU, DT = 2e5, 0.3, 1e-3


def _rotations(n, rng):
    q, r = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    q *= np.sign(np.diagonal(r, axis1=1, axis2=2))[:, None, :]
    q[np.linalg.det(q) < 0, :, 0] *= -1
    return q


def _stress(F, material, mu, lam):
    U, s, Vt = np.linalg.svd(F)
    if material == "sand":
        e = np.log(s)
        c = (2 * mu * e + lam * e.sum(1, keepdims=True)) / s
        return ((U * c[:, None, :]) @ Vt) @ F.transpose(0, 2, 1)
    J = np.linalg.det(F)
    return 2 * mu * (F - U @ Vt) @ F.transpose(0, 2, 1) + (lam * J * (J - 1))[:, None, None] * np.eye(3)


@pytest.mark.parametrize("material", ["sand", "jelly"])
@pytest.mark.parametrize("s_max, s_min", [(1.01, 0.99), (1.3, 0.77), (1.0, 0.38), (0.35, 0.3), (0.3, 0.2), (0.2, 0.12),
                                          (2.0, 0.15), (2.8, 1.0), (5.0, 0.2), (20.0, 0.2), (100.0, 0.5)])
def test_stress_error_over_strains(cuda, material, s_max, s_min):
    n = M ** 3
    rng = np.random.default_rng(5)
    base = np.stack(np.meshgrid(*[np.arange(M)] * 3, indexing="ij"), -1).reshape(-1, 3) * 5 + 2
    x = ((base + 1.37) / N).astype(np.float32)
    s = np.exp(rng.uniform(np.log(s_min), np.log(s_max), (n, 3)))
    s[:, 0], s[:, 2] = s_max, s_min
    F = (_rotations(n, rng) * s[:, None, :]) @ _rotations(n, rng).transpose(0, 2, 1)
    fd = (F - np.eye(3)).astype(np.float32)
    sim = MPM_Simulator_WARP(n, n_grid=N, device=str(cuda))
    sim.set_parameters(material=material, E=E, nu=NU, friction_angle=30.0, gravity=(0.0, 0.0, 0.0))
    one, zero = torch.ones(n, device=cuda), torch.zeros(n, 3, device=cuda)
    sim.load_x_initial_from_tensor(torch.from_numpy(x))
    sim.load_mass_from_tensor(one)
    sim.load_vol_from_tensor(one)
    sim.set_parameters(density=1.0)
    sim.load_uvF_from_tensor(zero, zero, torch.from_numpy(fd).to(cuda))
    sim.load_sample_particle_index_from_tensor(torch.arange(n, dtype=torch.int32))
    sim.p2g2p_reduced(0, DT)
    sim.check_status()
    got = sim.mpm_state.grid_v_in.double().cpu().numpy()
    assert np.array_equal(sim.engine.export(A.FIELD_F).cpu().numpy().reshape(n, 3, 3), fd + np.eye(3, dtype=np.float32))

    fx = x.astype(np.float64) * N - base
    w = np.stack([0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1) ** 2, 0.5 * (fx - 0.5) ** 2], -1)
    dw = np.stack([fx - 1.5, -2 * (fx - 1), fx - 0.5], -1)
    tau = _stress((fd + np.eye(3, dtype=np.float32)).astype(np.float64), material, E / 2 / (1 + NU),
                  E * NU / (1 + NU) / (1 - 2 * NU))
    err = np.zeros((n, 27, 3))
    ref = np.zeros((n, 27, 3))
    for q in range(27):
        a, b, c = q // 9, q // 3 % 3, q % 3
        grad = np.stack([dw[:, 0, a] * w[:, 1, b] * w[:, 2, c], w[:, 0, a] * dw[:, 1, b] * w[:, 2, c],
                         w[:, 0, a] * w[:, 1, b] * dw[:, 2, c]], -1)
        ref[:, q] = -DT * N * np.einsum("nrc,nc->nr", tau, grad)
        err[:, q] = got[base[:, 0] + a, base[:, 1] + b, base[:, 2] + c] - ref[:, q]
    rel = np.linalg.norm(err.reshape(n, -1), axis=1) / np.linalg.norm(ref.reshape(n, -1), axis=1)
    # near F = I the stress is as small as F - I, and F's own rounding counts relative to it
    strain = min(1.0, max(abs(np.log(s_max)), abs(np.log(s_min))))
    assert np.median(rel) <= 8.0 * 2.0 ** -24 * s_max / s_min / strain
