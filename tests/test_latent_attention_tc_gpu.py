"""Latent attention of portions of prompts on tcgen05 against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(q, z, rank, scale, positions, window):
    """q [n, heads, za], z [keys, za] float64 -> [n, heads, rank]."""
    s = torch.einsum("nhd,kd->nhk", q, z) * scale
    k = torch.arange(z.shape[0], device=z.device)
    hidden = k[None, :] > positions[:, None]
    if window:
        hidden |= k[None, :] <= positions[:, None] - window
    return torch.einsum("nhk,kd->nhd", torch.softmax(s.masked_fill(hidden[:, None], -torch.inf), -1), z[:, :rank])


# sequences: (tokens in the cache after the step, tokens of the step).  Tiles are 128 // heads queries by 64 keys: one token alone, whole
# tiles, one more and one less, a portion deep into its context, heads that leave rows over, one query a tile, single tokens deep into theirs
# beside a portion
@pytest.mark.parametrize("heads,rank,page,window,seqs", [
    (16, 512, 16, 0, [(1, 1), (64, 64), (65, 65), (63, 9), (200, 7)]),
    (16, 512, 32, 0, [(321, 130), (128, 128)]),
    (8, 256, 16, 0, [(1, 1), (127, 127), (129, 17), (700, 40)]),
    (12, 512, 64, 0, [(150, 21), (64, 1)]),
    (128, 256, 128, 0, [(130, 5), (3, 3)]),
    (16, 512, 16, 50, [(300, 60), (40, 40)]),
    (5, 256, 128, 64, [(260, 100)]),
    (16, 512, 16, 0, [(700, 1), (515, 1), (300, 77), (1100, 1), (64, 1)]),
    (8, 256, 64, 100, [(1000, 1), (333, 33), (129, 1)]),
])
def test_against_float64(heads, rank, page, window, seqs):
    from llmgen_b200.kernels import ops
    rot, za, dev = 64, rank + 64, "cuda"
    g = torch.Generator().manual_seed(heads * 1000 + rank + page + window)
    bq = ops.latent_attention_tc_tile_queries(torch.bfloat16, heads, rank, rot, page)
    assert bq == 128 // heads
    per_seq = max((c + page - 1) // page for c, _ in seqs)
    pages = torch.randperm(per_seq * len(seqs) + 1, generator=g)
    # what no sequence of this step has written holds no numbers
    cache = torch.full((len(pages), 1, page, za), torch.nan, dtype=torch.bfloat16)
    T = sum(n for _, n in seqs)
    q = torch.randn(T, heads, za, generator=g)
    tables, want, tiles, t = [], [], [], 0
    scale = za ** -0.5
    for i, (c, n) in enumerate(seqs):
        table = pages[i * per_seq:(i + 1) * per_seq].tolist()
        z = torch.randn(c, za, generator=g).to(torch.bfloat16)
        for k in range(c):
            cache[table[k // page], 0, k % page] = z[k]
        want.append(_exact(q[t:t + n].to(torch.bfloat16).double(), z.double(), rank, scale, torch.arange(c - n, c), window))
        if window:                                       # pages that the window has passed have been given back
            table = [-1 if (j + 1) * page <= c - n - window + 1 else p for j, p in enumerate(table)]
        tables += table
        tiles += [(i, a) for a in range(0, n, bq)]
        t += n
    tiles.append((-1, 0))                                # padding of a list of fixed length
    want = torch.cat(want).reshape(T, heads * rank)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    cu = [0]
    for _, n in seqs:
        cu.append(cu[-1] + n)
    common = (cache.to(dev), ints(tables), per_seq, ints([c for c, _ in seqs]), ints(cu), ints([a for a, _ in tiles]), ints([b for _, b in tiles]), T, heads,
              rank, rot, page, scale)
    out = torch.full((T, heads * rank), 9.0, device=dev)
    ops.latent_attention_tc(out, q.reshape(T, heads * za).to(dev), *common, window=window)
    torch.cuda.synchronize()
    ops.check_tc_errors(out.device)
    # scores: 36 sums of 16 products in float32, scale 1: about 4e-6; that moves a weight, and an output by its share of values of about 1
    assert float((out.cpu().double() - want).abs().max()) < 2e-5
    # head-major bfloat16 in and out: the same sums, rounded once
    pad = (T + 127) // 128 * 128
    q_hm = torch.zeros(heads, pad, za, dtype=torch.bfloat16, device=dev)
    q_hm[:, :T] = q.permute(1, 0, 2).to(torch.bfloat16)
    o_hm = torch.full((heads, pad, rank), 9.0, dtype=torch.bfloat16, device=dev)
    ops.latent_attention_tc(None, None, *common, out_head_major=o_hm, window=window, q_head_major=q_hm)
    assert torch.equal(o_hm[:, :T].permute(1, 0, 2).reshape(T, heads * rank), out.to(torch.bfloat16))
    assert bool((o_hm[:, T:] == 9.0).all())


def test_a_score_that_is_no_number_makes_its_row_none():
    from llmgen_b200.kernels import ops
    heads, rank, rot, page, T = 16, 512, 64, 16, 40
    dev, za = "cuda", 576
    g = torch.Generator().manual_seed(3)
    q = torch.randn(T, heads, za, generator=g)
    q[5, 3, 7] = torch.nan
    cache = torch.randn(3, 1, page, za, generator=g).to(torch.bfloat16).to(dev)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    out = torch.empty(T, heads, rank, device=dev)
    ops.latent_attention_tc(out, q.to(dev), cache, ints([0, 1, 2]), 3, ints([T]), ints([0, T]), ints([0] * 5), ints(range(0, T, 8)), T, heads, rank,
                            rot, page, za ** -0.5)
    lost = torch.isnan(out).all(-1).cpu()
    assert lost.nonzero().tolist() == [[5, 3]] and not bool(torch.isnan(out[~lost.to(dev)]).any())


def test_refusals():
    from llmgen_b200.kernels import ops
    bf = torch.bfloat16
    assert ops.latent_attention_tc_tile_queries(torch.float32, 16, 512, 64, 16) == 0
    assert ops.latent_attention_tc_tile_queries(bf, 129, 512, 64, 16) == 0
    assert ops.latent_attention_tc_tile_queries(bf, 16, 384, 64, 16) == 0
    assert ops.latent_attention_tc_tile_queries(bf, 16, 512, 32, 16) == 0
    assert ops.latent_attention_tc_tile_queries(bf, 16, 512, 64, 8) == 0
