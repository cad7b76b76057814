"""Rules of the instruction set that the compiler does not check, on the kernels' sources."""
import glob
import os
import re

import pytest

from foundry_b200.kernels.library import CSRC

# helpers of tcgen05.cuh whose instructions have cta_group::1
ONE_CTA = re.compile(r"\b(tc_commit|umma|umma_a_tmem)\(")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu"))), ids=os.path.basename)
def test_one_cta_group_in_all_tcgen05_instructions_of_a_kernel(path):
    """The allocation of tensor memory included. A file's kernels are of one kind here."""
    with open(path) as handle:
        text = re.sub(r"//[^\n]*", "", handle.read())
    groups = set(re.findall(r"tcgen05[a-z_.0-9]*\.cta_group::([12])", text))
    groups |= set(re.findall(r"cp\.async\.bulk\.tensor[a-z0-9_.]*\.cta_group::([12])", text))
    if ONE_CTA.search(text):
        groups.add("1")
    assert len(groups) <= 1, f"{os.path.basename(path)}: cta_group {sorted(groups)}"


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_an_aligned_cluster_barrier_meets_whole_warps(path):
    """`.aligned` wants the warp's lanes together, and the compiler does not bring them together again
    behind a branch or a loop: whoever issues the barrier does, right in front of it."""
    with open(path) as handle:
        text = re.sub(r"//[^\n]*", "", handle.read())
    for body in re.findall(r"\{[^{}]*barrier\.cluster\.arrive[a-z.]*\.aligned[^{}]*\}", text):
        assert "__syncwarp();" in body.split("barrier.cluster")[0], body
