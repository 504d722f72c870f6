"""What the kernels' sources keep to. Every kernel may start beside the kernel that writes its inputs (programmatic dependent launch)
and waits for it; the read-only path promises that nobody writes them while the kernel runs, so no load may take it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quantforge_b200", "csrc")
SOURCES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_load_through_the_read_only_path(path):
    with open(path) as f:
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)
    found = re.findall(r"\b__ldg\s*\(|\bld\.global\S*\.nc\b|\bconst\b[^;,(){}]*\*\s*(?:const\s+)?__restrict__", code)
    assert not found, found
