"""Kernels that start while the one before them still writes: no load of theirs takes the non-coherent path, which is
not held to the order of the wait.  Read from the sources: on the GPU a stale value would be a matter of luck."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flash_attn_with_score_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu*")))


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(f) for f in FILES])
def test_no_non_coherent_loads_beside_an_overlapped_launch(path):
    with open(path) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    if "griddep_wait" not in code:
        return
    found = re.findall(r"__ldg\s*\(|ld\.global\.nc|\bconst\s+\w+\s*\*\s*__restrict__", code)
    assert not found, found
