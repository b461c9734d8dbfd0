"""Warp-collective instructions (.aligned: tensor memory, cluster barriers) are issued
only by wrappers that converge the warp first: their callers store solutions under
per-lane conditions (systems past the batch, rows past a tail) right before, and a lane
still in such a branch leaves the instruction undefined.  Read from the sources, no GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "filtered_tdma_b200", "csrc")
FUNC = re.compile(r"^__device__ __forceinline__ [^;{]*\{\n(.*?)^\}", re.M | re.S)
ASM = re.compile(r'asm volatile\(\s*"[^"]*\.aligned')


def test_collectives_follow_a_converged_warp():
    found = 0
    for name in sorted(os.listdir(CSRC)):
        src = open(os.path.join(CSRC, name)).read()
        total = len(ASM.findall(src))
        wrapped = 0
        for body in FUNC.findall(src):
            n = len(ASM.findall(body))
            if n:
                wrapped += n
                assert body.lstrip().startswith("__syncwarp();"), (name, body)
                # nothing between them can part the lanes again
                assert not re.search(r"\b(if|for|while|switch)\b|\?", body), (name, body)
        assert wrapped == total, (name, "collective outside a wrapper")
        found += total
    assert found >= 8
