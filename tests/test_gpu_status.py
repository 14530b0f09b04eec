"""The lazy status word when the GPU lags behind the host: the fault of any
earlier substep is raised by the first call after the GPU has caught up, once."""
import pytest
import torch

from reduced_mpm_stress_training_gb300 import scenarios as S
from reduced_mpm_stress_training_gb300.engine import MPMStatusError

from helpers import gpu_sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lag", [False, True])
@pytest.mark.parametrize("before", [0, 1, 3])
def test_fault_is_raised_after_the_gpu_caught_up(cuda, before, lag):
    sc = S.small_column(64, 16)
    x0, v0, vol, mass = sc.particles()
    sim = gpu_sim(sc, x0=x0, v0=v0, vol=vol, mass=mass)
    good = torch.from_numpy(x0).to(cuda)
    bad = good.clone()
    bad[5] = 2.0  # outside the grid
    torch.cuda.synchronize()
    if lag:
        torch.cuda._sleep(200_000_000)  # a bounded wait on the stream (about 0.1 s)
    for k in range(before):
        sim.p2g2p(k, sc.dt)
    sim.load_x_initial_from_tensor(bad)  # on the device: does not wait for the GPU
    if not lag:
        torch.cuda.synchronize()
    for k in range(3 if lag else 1):
        sim.p2g2p(k, sc.dt)
    torch.cuda.synchronize()
    with pytest.raises(MPMStatusError):
        sim.p2g2p(9, sc.dt)
    sim.load_x_initial_from_tensor(good)
    sim.p2g2p(10, sc.dt)
    assert sim.check_status() == 0
    assert sim.engine.status() == 0
