"""The particle kernels of the adjoint move 36-word adjoint records as 16-byte
quads where the caller's buffers allow it and as words where a view starts at
another word: both give the same adjoint."""
import numpy as np
import pytest
import torch

from reduced_mpm_stress_training_gb300 import _capi as A
from reduced_mpm_stress_training_gb300 import scenarios as S
from reduced_mpm_stress_training_gb300.adjoint import SandRollout

pytestmark = pytest.mark.gpu

# Same arithmetic on the same saved forward; only the order of the float
# atomics into the grid adjoint differs: some 200 terms a node at 2**-24 each
# (1.2e-5) in the worst case, over two substeps.
TOL = 2.5e-5


@pytest.mark.parametrize("n", [1, 127, 129, 4000])
def test_buffers_at_any_word_give_the_same_adjoint(cuda, n):
    sc = S.small_column(n, 32, seed=5, floor_z=0.15, v0_sigma=0.1)
    sc.substeps = 2
    sand = SandRollout(sc, checkpoint_every=2, device=cuda)
    sand.forward(sand.v0_default, sc.E, sc.friction_angle)
    gen = torch.Generator(device=cuda).manual_seed(n)
    seed = torch.randn(n, A.ADJ_WORDS, device=cuda, generator=gen)
    words = n * A.ADJ_WORDS
    got = {}
    for offsets in ((0, 0), (1, 1), (0, 2)):
        sand.adj = [torch.full((words + 8,), 7.0, device=cuda)[o:o + words] for o in offsets]
        sand.backward(seed)
        got[offsets] = sand.state_bar[:, :33].double().cpu().numpy()
    fields = {"x": (0, 3), "v": (3, 6), "C": (6, 15), "F": (15, 24), "stress": (24, 33)}
    for offsets in ((1, 1), (0, 2)):
        for name, (a, b) in fields.items():
            want = got[(0, 0)][:, a:b]
            err = np.linalg.norm(got[offsets][:, a:b] - want)
            assert np.isfinite(want).all() and err <= TOL * np.linalg.norm(want), (offsets, name, err)
