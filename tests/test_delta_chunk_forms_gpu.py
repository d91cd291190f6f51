"""Both ways to a step's outputs of the chunked delta rule (csrc/head_delta.cu): in the walk for few chunks, side by side behind it."""
import pytest
import torch

from tests.plain import kugisun_plain as plain
from tests.test_kugisun_kernels_gpu import DEV, SIZES, close, memory_case, run_memory

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("behind", [False, True])
@pytest.mark.parametrize("H,G,D,E", SIZES)
def test_both_sides_of_the_line(H, G, D, E, behind):
    """Chunks that fill the SMs twice with their heads, and one place fewer: sequences at the edges of chunks among single tokens."""
    from llmgen_b200.kernels import ops
    line = (2 * ops.sm_count(torch.device(DEV)) + H - 1) // H
    lens = [130, 64, 65, 0, 1]
    places = lambda: sum(lens) // 64 + min(len(lens), sum(lens))
    if places() >= line:
        lens = [65, 1]
    while places() < line - (0 if behind else 1):
        lens.append(1 if places() + 1 < line else 0)
    assert places() == line - (0 if behind else 1)
    (q, k, v, beta, log_g), qkv, gates, state, cu, slots = memory_case(lens, H, G, D, E, 10)
    before = ops.launches()
    out, st = run_memory("chunks", qkv, gates, state, cu, slots, H, G, D, E)
    assert ops.launches() - before == (3 if behind else 2)
    for i in list(range(min(5, len(lens)))) + [len(lens) - 2]:
        a, b, S = cu[i], cu[i + 1], state[slots[i], :H * D * E].view(H, D, E).double()
        if lens[i]:
            o, S = plain.delta_memory(q[a:b].double(), k[a:b].double(), v[a:b].double(), beta[a:b].double(), log_g[a:b].double().exp(), S)
            close(out[a:b].view(lens[i], H, E), o, 3e-6)
        close(st[slots[i], :H * D * E].view(H, D, E), S, 3e-6)
    assert torch.equal(st[:, H * D * E:].cpu(), state[:, H * D * E:])
