"""Every `.aligned` barrier of the CUDA sources (and `bar.sync`, which is the aligned form) must be executed
by whole warps together, and code before it may have sent a warp's lanes apart: each is directly preceded by
__syncwarp().  Read from the sources, as a warp that is not together at such a barrier may hang the GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imps_cpp_tools_gb300", "csrc")
BARRIER = re.compile(r'asm volatile\(\s*"(barrier\.cluster\.(?:arrive|wait)[^"]*|bar\.sync[^"]*|'
                     r'tcgen05\.(?:alloc|dealloc)[^"]*)')


def barriers():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                text = f.read()
            for m in BARRIER.finditer(text):
                yield name, text[:m.start()], m.group(1)


def test_there_are_barriers():
    kinds = {b.split(".")[0] for _, _, b in barriers()}
    assert kinds == {"barrier", "bar", "tcgen05"}


@pytest.mark.parametrize("name", sorted({n for n, _, _ in barriers()}))
def test_whole_warps_at_aligned_barriers(name):
    for n, before, barrier in barriers():
        if n != name:
            continue
        lines = [re.sub(r"//.*", "", x).strip() for x in before.splitlines()]
        last = [x for x in lines if x][-1]
        assert last.endswith("__syncwarp();"), f"{name}: {barrier} after `{last}`"
