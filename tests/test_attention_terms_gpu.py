"""Causal attention with 32-bit softmax weights on the 5th-generation tensor cores at the edges of its tiles of 64 queries and 128 keys, against float64."""
import pytest
import torch

from llmgen_b200.kernels import build, ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HD = 128
SEQS = [(1, 1), (64, 64), (65, 65), (127, 3), (128, 128), (129, 1), (0, 2), (257, 200), (640, 65), (385, 385)]      # (context, new tokens); 0: padding


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("nq,nkv,page,sink,gate", [(2, 1, 16, None, None), (8, 2, 64, "values", "element"), (4, 2, 128, "zero", "head"), (12, 2, 32, None, "element")])
@pytest.mark.parametrize("sharp", [1.0, 12.0])
def test_causal_attention_with_exact_weights(nq, nkv, page, sink, gate, sharp):
    assert build.load("attention_tc").llmk_attention_tc_terms_usable(nq, nkv, HD, HD, page)
    T = sum(n for _, n in SEQS)
    most = max(-(-c // page) for c, _ in SEQS)
    pages = sum(-(-c // page) for c, _ in SEQS)
    # slots that no sequence owns hold no numbers: nothing may be read out of them, not even times zero
    kc, vc = (torch.full((pages, nkv, page, HD), float("nan"), dtype=torch.bfloat16) for _ in range(2))
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(1)).tolist()
    bt = torch.zeros(len(SEQS), most, dtype=torch.int32)
    q = rnd((T, nq, HD), 2, sharp)
    sinks = torch.randn(nq, generator=torch.Generator().manual_seed(3))
    gates = rnd((T, nq * HD if gate == "element" else nq), 4) if gate else None
    want, scale, cu, tiles = torch.zeros(T, nq, HD, dtype=torch.float64), HD ** -0.5, [0], []
    for s, (ctx, n) in enumerate(SEQS):
        own = [order.pop() for _ in range(-(-ctx // page))]
        bt[s, :len(own)] = torch.tensor(own, dtype=torch.int32)
        tiles += [(s, q0) for q0 in range(0, n, 64)]
        if ctx:
            k, v = rnd((ctx, nkv, HD), 10 + s), rnd((ctx, nkv, HD), 30 + s)
            for j in range(ctx):
                kc[own[j // page], :, j % page], vc[own[j // page], :, j % page] = k[j], v[j]
            k, v = (x.double().repeat_interleave(nq // nkv, 1) for x in (k, v))
            z = torch.einsum("thd,jhd->htj", q[cu[-1]:cu[-1] + n].double(), k) * scale
            hidden = torch.arange(ctx)[None, :] > torch.arange(ctx - n, ctx)[:, None]
            z = z.masked_fill(hidden[None], float("-inf"))
            if sink:
                extra = (sinks.double() if sink == "values" else torch.zeros(nq, dtype=torch.float64))[:, None, None].expand(nq, n, 1)
                p = torch.softmax(torch.cat([z, extra], 2), 2)[..., :ctx]
            else:
                p = torch.softmax(z, 2)
            want[cu[-1]:cu[-1] + n] = torch.einsum("htj,jhd->thd", p, v)
        cu.append(cu[-1] + n)
    if gate:
        want = want * torch.sigmoid(gates.double()).view(T, nq, -1)
    out = torch.full((T, nq * HD), 7.0, dtype=torch.bfloat16, device=DEV)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    ops.attention_mma(out, q.view(T, nq * HD).to(DEV), kc.to(DEV), vc.to(DEV), bt.to(DEV), most, ints([c for c, _ in SEQS]), ints(cu),
                      ints([t[0] for t in tiles] + [-1]), ints([t[1] for t in tiles] + [0]), len(tiles) + 1, nq, nkv, HD, HD, page, 0, scale, sink=sink is not None,
                      sink_values=sinks.to(DEV) if sink == "values" else None, gate=gates.to(DEV) if gate else None, gate_per_head=gate == "head")
    torch.cuda.synchronize()
    ops.check_tc_errors(out.device)
    got = out.cpu().double().view(T, nq, HD)
    # the result is rounded once to bfloat16, whose 8 significant bits put it at most 2^-8 of the value off.  Before that: a score is a float32 sum of 128 products of up to `sharp` times 4 sigma, good to
    # 128 2^-24 of their magnitudes' sum, and a weight's relative error is its score's error; sums over at most 640 keys add 640 2^-24.
    zmax = float((q.double().abs().sum(2).max() * 4.5) * scale)
    slack = (128 * zmax + 640) * 2.0 ** -24 * 2 * float(want.abs().max())
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + slack).all()), float(((got - want).abs() - want.abs() * 2.0 ** -8).max())
