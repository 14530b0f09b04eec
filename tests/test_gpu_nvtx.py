"""A profiler's timeline shows a substep's stages by name: the NVTX ranges of the library
as a tool sees them (a small one, compiled here and injected into a child process)."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

TESTS = os.path.dirname(os.path.abspath(__file__))
CHILD = """
import sys
sys.path[:0] = [{root!r}, {tests!r}]
from helpers import gpu_sim
from reduced_mpm_stress_training_gb300 import scenarios as S
sc = S.small_column(1000, 16)
sim = gpu_sim(sc)
sim.engine.ordered = {ordered}
sim.p2g2p(0, sc.dt)
sim.check_status()
"""


@pytest.mark.parametrize("ordered", [False, True])
def test_substep_stages_have_their_ranges(cuda, tmp_path, ordered):
    tool, names = tmp_path / "libnvtx_names.so", tmp_path / "names"
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["gcc", "-shared", "-fPIC", "-DNVTX_NO_IMPL", "-I", include, os.path.join(TESTS, "nvtx_names.c"),
                    "-o", str(tool)], check=True)
    env = dict(os.environ, NVTX_INJECTION64_PATH=str(tool), NVTX_NAMES=str(names))
    child = CHILD.format(root=os.path.dirname(TESTS), tests=TESTS, ordered=ordered)
    subprocess.run([sys.executable, "-c", child], env=env, check=True, timeout=120)
    substep, p2g = ("mpm_p2g2p_ordered", "mpm_p2g_ordered") if ordered else ("mpm_p2g2p", "mpm_p2g")
    lines = names.read_text().split("\n")
    at = lines.index(f"0 {substep}")
    assert lines[at + 1:at + 5] == [f"1 {n}" for n in ("mpm_sort", p2g, "mpm_grid_update", "mpm_g2p")]
