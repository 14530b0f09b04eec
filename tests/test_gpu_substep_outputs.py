"""All that one substep writes: mpm_p2g2p's own G2P form against the mpm_g2p stage (two
compilations that round differently), C and stress included, and a particle outside the
domain, whose record both forms carry over as it is.

Bounds on the root mean square error of a component, from the inputs and in units of
eps = 2^-24.  A node velocity is a sum of a few tens of terms: its error is taken as 16
eps |v|.  C = 4 / dx sum w g (i - fx) takes 27 products of weights below 1 and offsets
below 2 with it: 64 eps x 4 / dx x |v|.  The velocity gradient likewise, F_trial = (I + dt grad v) F:
dt 64 eps 4 / dx |v| + 8 eps.  The stress follows F_trial with at most 2 mu + 3 lam, twice
where the return map projects and twice for F away from I."""
import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S
from reduced_mpm_stress_training_gb300.engine import lame_from_E_nu

from helpers import gpu_sim, gpu_state

pytestmark = pytest.mark.gpu

GRID = 16
EPS = 2.0 ** -24


def _rms(a):
    return float(np.sqrt(np.mean(np.square(a, dtype=np.float64))))


@pytest.mark.parametrize("material", ["sand", "metal", "jelly"])
@pytest.mark.parametrize("chunk", [32, 64, 128, 256])
def test_every_field_of_both_forms(cuda, chunk, material):
    rng = np.random.default_rng(chunk)
    n = 3 * chunk + 37
    kw = dict(E=2e5, density=2000.0, yield_stress=2e3, hardening=1, xi=0.1) if material == "metal" else {}
    sc = S.small_column(n, GRID, material="metal" if material == "metal" else "sand", **kw)
    sc.material = material
    x0 = (rng.uniform(4.0, 13.4, (n, 3)) / GRID).astype(np.float32)
    x0[-1] = 1.5  # outside
    v = rng.normal(size=(n, 3)).astype(np.float32)
    F = (np.eye(3) + 0.02 * rng.normal(size=(n, 3, 3)) - 0.03 * np.eye(3)).astype(np.float32)
    C = rng.normal(size=(n, 3, 3)).astype(np.float32)
    tau = (100.0 * rng.normal(size=(n, 3, 3))).astype(np.float32)
    out = []
    for whole in (True, False):
        sim = gpu_sim(sc, chunk_size=chunk, x0=x0, v0=v, vol=np.full(n, 1e-5, np.float32),
                      mass=np.full(n, 2e-2, np.float32))
        sim.on_error = "ignore"
        e = sim.engine
        e.load(A.FIELD_C, torch.from_numpy(C))
        e.load(A.FIELD_F, torch.from_numpy(F))
        e.load(A.FIELD_STRESS, torch.from_numpy(tau))
        before = gpu_state(sim)
        if whole:
            e.substep_raw(0.0, sc.dt)
        else:
            for name in ("sort", "p2g", "grid", "g2p"):
                e.stage(name, time=0.0, dt=sc.dt)
            speed = float(e.export_grid(0)[2].abs().max())
        after = gpu_state(sim)
        for f in before:  # the particle outside
            assert np.array_equal(after[f][-1], before[f][-1]), f
        assert e.status() & A.ST_OUT_OF_DOMAIN
        e.clear_status()
        out.append(after)
    a, b = ({f: t[:-1] for f, t in o.items()} for o in out)
    dC = 64 * EPS * 4 * GRID * speed
    dF = sc.dt * dC + 8 * EPS
    mu, lam = lame_from_E_nu(sc.E, sc.nu)
    bounds = {"C": dC, "F": 2 * dF, "stress": 4 * (2 * mu + 3 * lam) * dF, "v": 32 * EPS * speed,
              "x": sc.dt * 32 * EPS * speed + 4 * EPS}
    if material == "metal":
        bounds["yield_"] = 4 * 2 * mu * dF
    for f, bound in bounds.items():
        assert np.isfinite(a[f]).all() and np.isfinite(b[f]).all(), f
        assert _rms(a[f] - b[f]) <= bound, (f, _rms(a[f] - b[f]), bound)
        assert _rms(b[f]) > 100 * bound or f == "yield_", (f, _rms(b[f]), bound)  # the bound says something
