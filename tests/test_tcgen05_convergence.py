"""The .aligned tensor-memory instructions are issued by whole warps: ahead of each load and
each release of tensor memory stands an instruction that brings the warp's lanes together,
with no loop entered in between (lanes that skip a store, or run out of a wait, fall behind)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cdixx_gb300" / "csrc"
FILES = [f.name for f in sorted(CSRC.glob("*.cu*")) if '"tcgen05.ld' in f.read_text() or '"tcgen05.dealloc' in f.read_text()]


def test_files_found():
    assert {"cdx_umma.cuh", "cdx_unet_umma.cuh", "cdx_fft.cuh"} <= set(FILES)


@pytest.mark.parametrize("name", FILES)
def test_aligned_instructions_follow_a_warp_barrier(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for m in re.finditer(r'"tcgen05\.(?:ld|dealloc)\.', text):
        joins = [j.end() for j in re.finditer(r"__syncwarp\(\);|__syncthreads\(\);", text[:m.start()])]
        between = text[joins[-1]:m.start()]
        assert not re.search(r"\b(?:for|while|continue|break|return)\b|mbar_\w+|_wait\w*\(", between), (name, between)
