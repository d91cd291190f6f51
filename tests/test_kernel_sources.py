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
