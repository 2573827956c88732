"""Rules of the CUDA sources that a compiler does not check."""
import glob
import os
import re

import pytest

from spikesorting_fullpursuit_b200 import build


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(build.CSRC, "*.cu*"))), ids=os.path.basename)
def test_inline_assembly_is_volatile(path):
    """Every piece here synchronises lanes, touches memory or waits: without `volatile` the
    compiler may drop it or move it into a branch that part of a warp takes."""
    with open(path) as fp:
        code = re.sub(r"//[^\n]*", "", fp.read())
    assert not re.findall(r"\basm\b(?!\s+volatile\b)", code)
