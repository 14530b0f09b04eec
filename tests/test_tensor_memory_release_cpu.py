"""After a tensor-core wait ran out, MMAs may still be writing tensor memory.  Every kernel
that releases tensor memory first gives the commit whose wait ran out another bounded
wait.  A wait flips the parity whether it ran out or not, so that commit has the parity
``phase ^ 1``; a wait for ``phase`` alone returns at once while it is pending (the phase
before it is complete).

No test can make a wait run out (that would be a hang), so this reads the sources, and
checks the parity rule on a model of an mbarrier of one arrival."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "reduced_mpm_stress_training_gb300",
                    "csrc")


class Mbarrier:
    """The PTX rule: try_wait.parity(p) is true when the current phase's parity is not p."""

    def __init__(self):
        self.completed = 0

    def arrive(self):
        self.completed += 1

    def try_wait(self, parity):
        return (self.completed & 1) != parity


def test_parity_of_the_commit_that_ran_out():
    for earlier in range(4):
        bar, phase = Mbarrier(), 0
        for _ in range(earlier):
            bar.arrive()
            assert bar.try_wait(phase)
            phase ^= 1
        assert not bar.try_wait(phase)  # runs out
        phase ^= 1
        assert bar.try_wait(phase)  # no wait at all
        assert not bar.try_wait(phase ^ 1)  # the commit that ran out
        bar.arrive()
        assert bar.try_wait(phase ^ 1) and not bar.try_wait(phase)  # then the one after it
        bar.arrive()
        assert bar.try_wait(phase)


def test_release_waits_for_the_commit_that_ran_out():
    releases = 0
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            src = re.sub(r"//[^\n]*", "", f.read())
        for m in re.finditer(r"tcgen05\.dealloc", src):
            releases += 1
            kernel = src[max(src.rfind("__global__", 0, m.start()), src.rfind("void tc_teardown", 0, m.start())):m.start()]
            assert re.search(r"mbar_wait\((&s\.)?mbar, phase \^ 1u\);", kernel), os.path.basename(path)
    assert releases == 4
