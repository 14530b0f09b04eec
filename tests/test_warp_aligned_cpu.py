"""Warp-wide (.aligned) tcgen05 and barrier instructions are undefined when the lanes of a
warp are not together.  The hand-written ones follow loops that lanes leave one by one
(mbarrier polls) and branches on the lane, so in the source each has to be preceded by
__syncwarp() or by another such instruction; where a caller brings the lanes together
itself, it has to do so behind each poll and before its loop over the layers."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "reduced_mpm_stress_training_gb300",
                    "csrc")
ASM = re.compile(r'asm volatile\((?:[^;"]|"(?:[^"\\]|\\.)*")*\);')


def _sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            yield os.path.basename(path), re.sub(r"//[^\n]*", "", f.read())


def test_lanes_are_together_before_warp_wide_tcgen05():
    seen = 0
    for name, src in _sources():
        ends = set()
        for m in ASM.finditer(src):
            if not re.search(r"tcgen05\.[\w:.]*\.sync\.aligned", m.group(0)):
                continue
            seen += 1
            before = src[:m.start()].rstrip()
            assert re.search(r"(^|\s)__syncwarp\(\);$", before) or len(before) in ends, (name, m.group(0)[:80])
            ends.add(m.end())
    assert seen >= 14  # allocations with their permits, loads with their waits, releases


def test_lanes_are_together_before_named_barriers():
    seen = 0
    for name, src in _sources():
        for m in ASM.finditer(src):
            if not re.search(r'"[^"]*(?:\\n|\b)bar\.(?:sync|red)\b', m.group(0)):
                continue
            seen += 1
            at = src.rindex("__device__", 0, m.start())
            if src[at:m.start()].split("(")[0].endswith(" pipe_barrier"):  # the caller's part, below
                continue
            assert "__syncwarp();" in src[at:m.start()], (name, m.group(0)[:80])
    assert seen >= 7


def test_a_caller_that_vouches_for_its_lanes():
    calls = 0
    for name, src in _sources():
        for m in re.finditer(r"tmem_ld32<true>\(", src):
            calls += 1
            poll = src.rindex("mbar_wait(", 0, m.start())
            assert "__syncwarp();" in src[poll:m.start()], name
        for m in re.finditer(r"\bpipe_barrier\(pipe\);", src):
            calls += 1
            loop = src.rindex("for (int layer", 0, m.start())
            assert src[:loop].rstrip().removesuffix("#pragma unroll 1").rstrip().endswith("__syncwarp();"), name
            # the loop's own branches on the lane: Z of rows past n
            body = src[loop:src.index("if (!ok) break;", loop)]
            assert body.count("if (io.z) __syncwarp();") == body.count("activate_chunk("), name
    assert calls >= 3
