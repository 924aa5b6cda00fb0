"""The library's streams are non-blocking ones, which wait for nothing on the default stream: no copy,
fill or launch in its sources goes there (a copy from pageable memory may return before its transfer
ends, and a kernel on another stream then reads what was there before)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cupdlp.jl_gb300", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.h")))


def _code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_everything_on_a_stream(path):
    code = _code(path)
    assert not re.findall(r"\bcuda(?:Memcpy|Memset|Memcpy2D|MemcpyToSymbol|MemcpyFromSymbol)\s*\(", code)
    for launch in re.findall(r"<<<(.*?)>>>", code, flags=re.S):
        depth, parts = 0, 1
        for ch in launch:
            depth += ch in "([{"
            depth -= ch in ")]}"
            parts += ch == "," and depth == 0
        assert parts == 4, launch   # grid, block, shared memory, stream


def test_streams_are_non_blocking():
    calls = [c for p in SOURCES for c in re.findall(r"cudaStreamCreate\w*\(([^;]*)\)", _code(p))]
    assert calls and all("cudaStreamNonBlocking" in c for c in calls)
