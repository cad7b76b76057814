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


def kernels_of(name):
    """The kernels of a source file: name -> text."""
    with open(os.path.join(CSRC, name)) as handle:
        text = re.sub(r"//[^\n]*", "", handle.read())
    found = {}
    for part in text.split("__global__")[1:]:
        body = part[:part.index("\n}\n")]
        found[re.search(r"(\w+_kernel)\s*\(", body).group(1)] = body
    return found


def test_what_writes_states_lets_nobody_start_before():
    """The single-token kernels ask for the state before they wait for the kernel in front: nobody who
    writes states may let a successor start early. The kernels of a state are those that know its place."""
    kernels = {}
    for name in ("sequence_mix.cu", "chunk_scan.cu", "linear_step.cu", "state_step.cu", "elementwise.cu"):
        kernels.update(kernels_of(name))
    of_states = {n for n, body in kernels.items() if "s_offset" in body} | {"zero_rows_kernel", "linear_chunk_kernel"}
    assert {"scan_kernel", "walk_kernel", "linear_step_kernel", "state_step_kernel"} <= of_states <= set(kernels)
    for name in of_states:
        body = kernels[name]
        if name == "linear_step_kernel":  # behind its writes
            early, body = body.split("fb_pdl_launch();")
            assert "reinterpret_cast<float4*>(S" in early and not re.search(r"\(S \+[^;]*\) = ", body)
        assert "fb_pdl_launch" not in body, name


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))), ids=os.path.basename)
def test_an_aligned_cluster_barrier_meets_whole_warps(path):
    """`.aligned` wants the warp's lanes together, and the compiler does not bring them together again
    behind a branch or a loop: whoever issues the barrier does, right in front of it."""
    with open(path) as handle:
        text = re.sub(r"//[^\n]*", "", handle.read())
    for body in re.findall(r"\{[^{}]*barrier\.cluster\.arrive[a-z.]*\.aligned[^{}]*\}", text):
        assert "__syncwarp();" in body.split("barrier.cluster")[0], body
