"""Contracts of the kernels that a run on a healthy GPU cannot show and must not be made to show, read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kandle_b200", "csrc")


def _code(path):
    """The source without its comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)


@pytest.mark.parametrize("name", sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu*"))))
def test_aligned_cluster_barriers_follow_a_reconvergence(name):
    """barrier.cluster with .aligned needs all lanes of a warp at the same instruction; roles that end at different times
    do not give that by themselves."""
    code = _code(os.path.join(CSRC, name))
    for m in re.finditer(r'asm volatile\(\s*"barrier\.cluster\.arrive[^"]*\.aligned', code):
        assert re.search(r"__syncwarp\(\);\s*$", code[:m.start()]), f"{name}: line {code[:m.start()].count(chr(10)) + 1}"
