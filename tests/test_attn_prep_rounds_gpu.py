"""q, k and v prepared in float32 with two and with four rounds of rows a warp (csrc/attn_prep.cu), at both sides of the line between them."""
import pytest
import torch

from tests.test_kernels_gpu import _attn_prep_on_prompts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("nq,nkv,hd", [(24, 12, 32), (24, 12, 64), (32, 8, 128), (3, 3, 128)])
def test_rows_at_both_sides(nq, nkv, hd, more):
    from llmgen_b200.kernels import ops
    line = 128 * 16 * ops.sm_count(torch.device("cuda:0")) // ((nq + 2 * nkv) * (hd // 8))
    _attn_prep_on_prompts(ops, torch.float32, nq, nkv, hd, line + more)
