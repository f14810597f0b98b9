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


@pytest.mark.parametrize("name", ["gemm_f32_split.cu", "recurrence.cuh"])
def test_whole_warps_give_up_together(name):
    """A wait that runs out for some lanes only would leave the others at the warp's next full-mask instruction.  Waits of
    whole warps are combined; the rest belong to one lane (`issue`, the copying warp's `lane == 0`)."""
    lines = _code(os.path.join(CSRC, name)).split("\n")
    for i, line in enumerate(lines):
        if "mbar_wait(" in line and "__all_sync(0xffffffffu" not in line:
            before = "\n".join(lines[:i])
            alone = max(before.rfind("auto issue = [&]()"), before.rfind("if (lane == 0) {"))
            warp_role = max(before.rfind("regs_inc<"), before.rfind("const int j = lane % LPC"))
            assert alone > warp_role, f"{name}: {line.strip()}"


def test_the_copying_warp_outlives_its_copies():
    """recurrence_kernel: consumers may give up after the copying warp's last request, so its wait for what is in flight
    may not hang on the abort flag of that moment."""
    code = _code(os.path.join(CSRC, "recurrence.cuh"))
    role = code[code.index("if (warp == consumers) {"):code.index("const int j = lane % LPC")]
    assert "mbar_try_wait(&full[s]" in role and "abort_flag)\n" not in role[role.rindex("bulk_load"):]
