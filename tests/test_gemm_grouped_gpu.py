"""The experts' products with swapped operands, and the runs of rows that they take, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plan(ops, counts):
    """Slots of experts with these many rows each: (order, spans)."""
    E = len(counts)
    slots = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).to(torch.int32)
    slots = slots[torch.randperm(len(slots), generator=torch.Generator().manual_seed(1))].cuda()
    n, tiles = len(slots), ops.moe_max_tiles(len(slots), E, 128)
    ints = lambda k: torch.full((k,), -7, dtype=torch.int32, device="cuda")
    order, pos, spans = ints(tiles * 128), ints(n), ints(4 * (ops.moe_max_spans(n, E) + 1))
    ops.moe_plan(slots, n, E, order, pos, ints(tiles), ints(tiles), ints(tiles), tile=128, padded=True, spans=spans)
    return slots, order, spans


# one row, a span's edges (255 .. 257, 32 .. 33), experts without rows, several spans of one expert
COUNTS = [[1], [0, 31, 32, 33, 0, 255, 256, 257, 0], [700, 1, 64, 513]]


@pytest.mark.parametrize("counts", COUNTS)
def test_spans(counts):
    from llmgen_b200.kernels import ops
    slots, order, spans = _plan(ops, counts)
    spans, order, slots = spans.view(-1, 4).tolist(), order.tolist(), slots.tolist()
    n = spans[0][0]
    assert n == sum((c + 255) // 256 for c in counts)
    seen = []
    for e, start, rows, width in spans[1:1 + n]:
        assert 0 < rows <= width <= 256 and width % 32 == 0
        assert all(slots[order[i]] == e for i in range(start, start + rows))
        seen += order[start:start + rows]
    assert sorted(seen) == list(range(len(slots)))


@pytest.mark.parametrize("activation,out_dtype", [(None, torch.float32), (None, torch.bfloat16), ("relu2", torch.bfloat16),
                                                  ("silu_glu", torch.bfloat16), ("clamped_glu", torch.bfloat16)])
@pytest.mark.parametrize("counts,N,K", [([1], 64, 64), (COUNTS[1], 288, 136), (COUNTS[2], 544, 1024), ([3, 2, 0, 9], 2048, 72)])
def test_against_float64(counts, N, K, activation, out_dtype):
    from llmgen_b200.kernels import ops
    from llmgen_b200.parts.mlp import interleave_gate_up
    E = len(counts)
    _, order, spans = _plan(ops, counts)
    g = torch.Generator().manual_seed(N + K + E)
    n = order.numel()
    x = torch.randn(n, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, N, K, generator=g) * 0.2).to(torch.bfloat16)
    rows = order >= 0
    x[~rows.cpu()] = torch.nan                            # rows of the padded order that nobody owns hold no numbers
    expert = torch.full((n,), -1, dtype=torch.long)
    for e, start, k, _ in spans.view(-1, 4).tolist()[1:1 + int(spans[0])]:
        expert[start:start + k] = e
    gated = activation in ("silu_glu", "clamped_glu")
    packed = torch.stack([interleave_gate_up(m[:N // 2], m[N // 2:]) for m in w]) if gated else w
    out = torch.full((n, N // 2 if gated else N), 7.0, dtype=out_dtype, device="cuda")
    ops.gemm_grouped(out, x.cuda(), packed.contiguous().cuda(), spans, activation, alpha=1.702, limit=4.0)
    torch.cuda.synchronize()
    ops.check_tc_errors(out.device)
    live = expert >= 0
    assert torch.equal(live, rows.cpu()) and bool((out.cpu()[~live] == 7.0).all())
    c = torch.stack([x[i].double() @ w[expert[i]].double().t() for i in live.nonzero().flatten().tolist()])
    if activation == "relu2":
        c = c.clamp(min=0) ** 2
    elif gated:
        a, u = c[:, :N // 2], c[:, N // 2:]
        if activation == "clamped_glu":
            a, u = a.clamp(max=4.0), u.clamp(-4.0, 4.0)
            c = a * torch.sigmoid(1.702 * a) * (u + 1)
        else:
            c = a * torch.sigmoid(a) * u
    err = float((out.cpu()[live].double() - c).abs().max())
    # float32 sums of K products; a bfloat16 result is rounded once (up to 2^-8 of it)
    assert err < (2e-5 if out_dtype == torch.float32 else 4e-3) * max(1.0, float(c.abs().max()))


def test_refusals():
    from llmgen_b200.kernels import ops
    x, w = torch.zeros(128, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(2, 48, 64, dtype=torch.bfloat16, device="cuda")
    spans = torch.zeros(16, dtype=torch.int32, device="cuda")
    with pytest.raises(ops.KernelError, match="multiple of 32"):
        ops.gemm_grouped(torch.zeros(128, 24, dtype=torch.bfloat16, device="cuda"), x, w, spans, "silu_glu")
    with pytest.raises(ops.KernelError, match="bfloat16 results"):
        ops.gemm_grouped(torch.zeros(128, 48, device="cuda"), x, w, spans, "relu2")
    with pytest.raises(ops.KernelError, match="not built"):
        ops.gemm_grouped(torch.zeros(128, 48, device="cuda"), x, w, spans, "tanh")
