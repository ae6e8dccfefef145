"""Kernels launched as programmatic dependents start before the kernels ahead of them have finished, so no tile may be
loaded before griddepcontrol.wait (only prefetched into L2): checked on the sources, since a missing wait rarely shows."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "sglang_b200", "csrc")
KERNELS = ["gemm_skinny.cuh", "linear_stream.cuh", "gemm_stream.cuh", "gemm_pair.cuh", "gemm_ue8m0.cuh", "gemm_ue8m0_pair.cuh",
           "gemm_kernel.cuh"]
WAIT = r"grid_dependency_wait\(\)|griddepcontrol\.wait"


@pytest.mark.parametrize("name", KERNELS)
def test_producer_loads_after_the_wait(name):
    text = open(os.path.join(CSRC, name)).read()
    body = text[text.index("__global__"):]
    # the TMA producer's branch: the elected thread of the producer warp, up to the next role
    role = re.search(r"if \(warp == (?:Cfg::)?kProducerWarp\) \{\s*(?:asm[^;]*;\s*)?if \(ptx::elect_one\(\)\)", body)
    assert role, "no producer branch found"
    branch = body[role.start():]
    branch = branch[:branch.index("else if (warp ==")]
    load = re.search(r"(?:tma_load_2d\w*|wide_load<\w+>)\(", branch)
    assert load, "no load found"
    # a wait of all warps before the roles part: unconditional, for the one mode that is launched as a dependent, or in
    # both branches of the stage
    waits, header = [], ""
    for line in body[:role.start()].splitlines():
        if re.match(r" {2}\S", line):
            header = line.split("//")[0].strip()
        if re.match(r" {2,4}(?:" + WAIT + ")", line):
            waits.append("all" if re.match(r" {2}\S", line) else header)
    everyone = "all" in waits or "if (MODE == GEMM_DENSE) {" in waits or \
        ("if (STAGE == STREAM_GATE_UP) {" in waits and "} else {" in waits)
    assert everyone or re.search(WAIT, branch[:load.start()]), "a tile is loaded before griddepcontrol.wait"
