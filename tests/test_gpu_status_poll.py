"""Reading the lazy status word after the GPU lagged: the read waits for nothing that
was queued behind the substep, and clearing the state does not lose a fault."""
import pytest
import torch

from reduced_mpm_stress_training_gb300 import scenarios as S
from reduced_mpm_stress_training_gb300.engine import MPMStatusError

from helpers import gpu_sim

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def loaded(cuda):
    """Every kernel loaded before a test: the host does not stop at a first launch."""
    sc = S.small_column(64, 16)
    sim = gpu_sim(sc)
    sim.p2g2p(0, sc.dt)
    sim.check_status()


def _lagging_steps(cuda, fault):
    """A simulator whose second substep was queued before the first had run."""
    sc = S.small_column(64, 16)
    x0, v0, vol, mass = sc.particles()
    if fault:
        x0[5] = 2.0  # outside the grid
    sim = gpu_sim(sc, x0=x0, v0=v0, vol=vol, mass=mass)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # a bounded wait on the stream (about 0.1 s)
    for k in range(2):
        sim.p2g2p(k, sc.dt)
    return sim, sc


@pytest.mark.parametrize("other_stream", [False, True])
@pytest.mark.parametrize("fault", [False, True])
def test_poll_does_not_wait_for_later_work(cuda, fault, other_stream):
    for _ in range(2):  # the second time with everything loaded
        sim, sc = _lagging_steps(cuda, fault)
        torch.cuda.synchronize()
        stream = torch.cuda.Stream(cuda) if other_stream else torch.cuda.current_stream(cuda)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_000_000_000)  # bounded: about half a second
            done = torch.cuda.Event()
            done.record()
            if fault:
                with pytest.raises(MPMStatusError):
                    sim.engine.poll_status()
            else:
                assert sim.engine.poll_status() == 0
            assert not done.query(), "poll_status waited for work queued after the substep"
        torch.cuda.synchronize()
        assert sim.engine.status() == 0
        assert sim.engine.poll_status() == 0


def test_reinit_keeps_an_unread_fault(cuda):
    sim, sc = _lagging_steps(cuda, True)
    sim.engine.reinit()
    torch.cuda.synchronize()
    with pytest.raises(MPMStatusError):
        sim.engine.poll_status()
    assert sim.engine.poll_status() == 0
