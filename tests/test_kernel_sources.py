"""What the kernels' sources keep to. Every kernel may start beside the kernel that writes its inputs (programmatic dependent launch)
and waits for it; the read-only path promises that nobody writes them while the kernel runs, so no load may take it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quantforge_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_load_through_the_read_only_path(path):
    code = _code(path)
    found = re.findall(r"\b__ldg\s*\(|\bld\.global\S*\.nc\b|\bconst\b[^;,(){}]*\*\s*(?:const\s+)?__restrict__", code)
    assert not found, found


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_what_one_lane_acquires_is_passed_on(path):
    """One lane polls a counter for its warp, inside a vote. Votes order no memory, so before the lanes' proxy fences, behind which they
    issue copies of what the counter guards, comes a warp barrier."""
    code = _code(path)
    for poll in re.finditer(r"lane\s*!=\s*0\s*\|\|\s*\w*acquire\w*\s*\(", code):
        fence = code.find("fence.proxy.async", poll.end())
        assert fence < 0 or "__syncwarp()" in code[poll.end():fence]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_warps_are_together_at_aligned_cluster_barriers(path):
    """The aligned forms are undefined for a warp whose threads are apart, as they may be behind any condition: each stands in a wrapper
    that brings them together first."""
    for asm in re.finditer(r'asm volatile\(\s*"barrier\.cluster\.[^"]*\.aligned', _code(path)):
        body = _code(path)[:asm.start()].rpartition("{")[2]
        assert "__syncwarp();" in body, body


def test_warps_are_together_at_loads_of_accumulators():
    """Where a warp's share of the columns may be cut short, its partial sums are stored under a condition that splits the warp, and the
    next load of accumulators is a whole warp's."""
    code = _code(os.path.join(CSRC, "qf_gemm_tcgen05.cu"))
    loop = code[code.index("for (int c8 = 0;"):code.index("__stcg(part")]
    assert "n < p.N" in loop and loop.index("if constexpr (RAGGED) __syncwarp();") < loop.index("tmem_ld8")
