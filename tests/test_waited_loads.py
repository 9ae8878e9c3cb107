"""Cycle kernels may be launched before the one ahead has ended: each waits first
(follow_on), and reads through the non-coherent path (__ldg) only what no kernel of the
cycle writes."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lulesh_gb300",
                    "csrc")
FILES = ["lg_kernels.cuh", "lg_kernels_lanes.cuh", "lg_kernels_team.cuh", "lg_kernels_mixed.cu"]


@pytest.mark.parametrize("name", FILES)
def test_kernels_wait_first_and_read_fields_coherently(name):
    src = open(os.path.join(CSRC, name)).read()
    kernels = re.findall(r"__global__[^{;]*?(k_\w+)\(DevState s\)\s*\{\s*([^;]*;)", src)
    assert kernels
    for kernel, first in kernels:
        assert first.strip() == "follow_on();", kernel
    reads = re.findall(r"__ldg\(&?([^\[)]*)", src)
    assert set(reads) <= {"s.nodelistT"}, reads
