"""Barrier instructions of the aligned kind (barrier.cluster ... .aligned, bar.sync) are undefined in a
warp whose lanes have not come together: every one in the device sources stands right behind a
__syncwarp()."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cupdlp.jl_gb300", "csrc")
ASM = re.compile(r'asm\s+volatile\s*\(\s*"[^"]*(?:\.aligned|bar\.sync|barrier\.sync)[^"]*"')


def _sources():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu*")))


@pytest.mark.parametrize("path", _sources(), ids=os.path.basename)
def test_warp_converges_first(path):
    text = open(path).read()
    for hit in ASM.finditer(text):
        before = re.sub(r"//[^\n]*", "", text[:hit.start()]).rstrip()
        assert before.endswith("__syncwarp();"), f"{os.path.basename(path)}: {hit.group(0)}"


def test_finds_the_cluster_barriers():
    assert sum(len(ASM.findall(open(p).read())) for p in _sources()) >= 2
