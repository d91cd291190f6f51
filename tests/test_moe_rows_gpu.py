"""The routed feed-forward's kernels for many tokens at the edges of what they take: the router's sixteen-token blocks, the plan's tiles, whole-vector
rows, the sums over slots."""
import pytest
import torch

from llmgen_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}


def rnd(shape, seed, scale=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n,E,K,top,gate", [(888, 8, 64, 2, False), (1185, 32, 1024, 4, True), (1200, 33, 1032, 3, False), (1199, 70, 2056, 8, True), (2050, 3, 8, 3, False)])
def test_the_router_over_many_tokens(n, E, K, top, gate, dtype):
    wide = rnd((n, K + 8), 1, 1.0, DT[dtype])
    h, router, bias = wide[:, :K], rnd((E + int(gate), K), 2, K ** -0.5), rnd((E,), 3)
    expert, weight = torch.full((n * top,), -7, dtype=torch.int32, device=DEV), torch.zeros(n * top, device=DEV)
    out = torch.zeros(n, device=DEV) if gate else None
    ops.moe_route(wide.to(DEV)[:, :K], router.to(DEV), expert, weight, top, "sigmoid", False, bias=bias.to(DEV), gate_out=out)
    z = h.double() @ router.double().T
    # a float32 sum: each of a chain's K / 8 additions, of the eight warps' and of the bias's rounds at most the sum of the magnitudes; a sigmoid's slope
    # is at most 1/4, and the function itself is good to a few units in the last place
    tol = float((K / 8 + 10) * 2.0 ** -24 * (h.double().abs() @ router.double().abs().T + 4).max()) / 4 + 4 * 2.0 ** -24
    if gate:
        assert float((out.cpu().double() - torch.sigmoid(z[:, E])).abs().max()) <= tol
    s = torch.sigmoid(z[:, :E] + bias.double())
    expert, weight = expert.view(n, top).cpu().long(), weight.view(n, top).cpu().double()
    assert int(expert.min()) >= 0 and int(expert.max()) < E and all(len(set(row)) == top for row in expert.tolist())
    assert float((weight - s.gather(1, expert)).abs().max()) <= tol
    assert float((weight - s.sort(1, descending=True).values[:, :top]).abs().max()) <= 2 * tol       # (experts may change places in a close call)


@pytest.mark.parametrize("n_slots,E,tile,padded", [(1, 5, 128, True), (130, 1, 128, True), (127, 33, 16, False), (8192, 32, 128, True), (8195, 33, 128, True),
                                                   (20001, 100, 128, True), (20001, 100, 16, False), (9000, 3, 128, True)])
def test_the_plan_gives_every_slot_one_row_of_its_expert(n_slots, E, tile, padded):
    expert = torch.randint(0, E + 2, (n_slots,), generator=torch.Generator().manual_seed(5))          # the last two have no products
    expert[expert == E // 2] = 0                                                                       # and one no slots
    tiles = ops.moe_max_tiles(n_slots, E, tile)
    order = torch.full((tiles * tile if padded else n_slots,), -9, dtype=torch.int32, device=DEV)
    pos, te, ts, tr = (torch.full((m,), -9, dtype=torch.int32, device=DEV) for m in (n_slots, tiles, tiles, tiles))
    ops.moe_plan(expert.to(torch.int32).to(DEV), n_slots, E, order, pos, te, ts, tr, tile=tile, padded=padded)
    order, pos, te, ts, tr = (v.tolist() for v in (order, pos, te, ts, tr))
    owner, want, at = {}, [], 0
    for e in range(E):
        count = int((expert == e).sum())
        for r in range(0, count, tile):
            want.append((e, at + r, min(tile, count - r)))
        for r in range(count):
            owner[at + r] = e
        at += -(-count // tile) * tile if padded else count
    assert [(e, s, r) for e, s, r in zip(te, ts, tr) if e >= 0] == want
    assert all(e == -1 and r == 0 for e, r in zip(te[len(want):], tr[len(want):]))
    for i in range(n_slots):
        e = int(expert[i])
        if e < E:
            assert order[pos[i]] == i and owner[pos[i]] == e
        else:
            assert pos[i] == -1
    if padded:
        assert sum(o >= 0 for o in order) == int((expert < E).sum()) and min(order) >= -1


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("K", [8, 256, 264, 2056, 12])
def test_rows_are_gathered_and_added_up(K, dtype):
    dt, n, top = DT[dtype], 19, 5
    wide, weight = rnd((n, K + 8), 1, 1.0, dt), rnd((n * top,), 2)
    order = torch.randperm(n * top, generator=torch.Generator().manual_seed(3)).to(torch.int32)
    order[::7] = -1
    for scaled in (False, True):
        out = torch.full((n * top, K), 7.0, dtype=dt, device=DEV)
        ops.moe_gather(out, wide.to(DEV)[:, :K], order.to(DEV), weight.to(DEV), top, scaled)
        rows = wide[:, :K].float()[order.clamp(min=0).long() // top] * (weight[order.clamp(min=0).long()][:, None] if scaled else 1.0)
        assert torch.equal(out.cpu(), torch.where(order[:, None] >= 0, rows, torch.full_like(rows, 7.0)).to(dt))
    rows = rnd((n * top, K), 4)
    for t in (1, 3, 4, 5):
        pos = torch.randperm(n * top, generator=torch.Generator().manual_seed(t))[:n * t].to(torch.int32)
        pos[::5] = -1                                                                                  # no row, no identity: nothing is added
        got = torch.empty(n, K, device=DEV)
        ops.moe_combine(got, rows.to(DEV), pos.to(DEV), None, t, slot_weight=weight[:n * t].to(DEV))
        terms = torch.where(pos[:, None] >= 0, rows[pos.clamp(min=0).long()].double() * weight[:n * t].double()[:, None], torch.zeros(1, dtype=torch.float64))
        bound = terms.abs().view(n, t, K).sum(1) * (t + 1) * 2.0 ** -24
        assert bool(((got.cpu().double() - terms.view(n, t, K).sum(1)).abs() <= bound).all())


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("E,K,top,gate,scoring", [(32, 2048, 4, False, "sigmoid"), (33, 1032, 3, True, "softmax"), (8, 72, 2, False, "sigmoid"), (70, 520, 8, True, "sigmoid")])
def test_a_tokens_experts_do_not_depend_on_how_many_tokens_share_the_step(E, K, top, gate, scoring, dtype):
    """The same bits whichever kernel takes the step: one token a block, four, sixteen."""
    n = 1190
    h, router, bias = rnd((n, K), 1, 1.0, DT[dtype]).to(DEV), rnd((E + int(gate), K), 2, K ** -0.5).to(DEV), rnd((E,), 3).to(DEV)

    def route(rows):
        m = len(rows)
        expert, weight, out = torch.full((m, top), -7, dtype=torch.int32, device=DEV), torch.zeros(m, top, device=DEV), torch.zeros(m, device=DEV)
        ops.moe_route(rows, router, expert.view(-1), weight.view(-1), top, scoring, False, bias=bias, gate_out=out if gate else None)
        return expert, weight, out
    whole = route(h)
    for size in (1, 37, 601):
        parts = [route(h[i:i + size]) for i in range(0, n if size > 1 else 20, size)]
        for got, want in zip(zip(*parts), whole):
            got = torch.cat(got)
            assert torch.equal(got, want[:len(got)])
