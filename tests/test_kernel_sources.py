"""What every kernel's source has to keep to under programmatic dependent launch (csrc/common.cuh)."""
import glob
import os
import re

import pytest

from tests.util import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "llmgen_b200", "csrc", "*.cu")) + glob.glob(os.path.join(ROOT, "llmgen_b200", "csrc", "*.cuh")))


def code(path):
    """The file without its comments."""
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_array_is_promised_to_stay_as_it_is(path):
    """The kernel before writes a kernel's inputs while its blocks are resident, and q, k, v are prepared in place: loads that the
    compiler may take for those of constant data could be moved in front of the wait.  Weights and the step's tables alone, which no
    kernel of a step writes, are read through the read-only path by name."""
    src = code(path)
    assert "__restrict__" not in src
    allowed = {"gemm_rows8.cu": ["ld.global.nc.v4.u32"], "moe.cu": ["__ldg(reinterpret_cast<const float4*>(w + k"]}
    for use in re.findall(r"ld\.global\.nc[.\w]*|__ldg\([^)]*", src):
        assert use in allowed.get(os.path.basename(path), []) or use.startswith("__ldg(bt + "), use


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_the_next_kernel_is_let_go_behind_the_allocation_of_tensor_memory(path):
    """A block of the next kernel that got its tensor memory first would wait for this kernel, which would wait for the tensor memory:
    an allocation has no limit on its wait."""
    for kernel in code(path).split("__global__")[1:]:
        body = kernel[:kernel.find("\n}\n")]
        if "tmem_alloc" in body and "pdl_launch_dependents()" in body:
            alloc = max(body.find("tmem_alloc("), body.find("tmem_alloc_pair("))
            ready = body.find("*tmem_slot;", alloc)             # read behind the barrier that follows the allocation
            assert 0 <= alloc < ready < body.find("pdl_launch_dependents()")
