"""Causal attention with 32-bit softmax weights on the 5th-generation tensor cores beside the same on `mma.sync` (csrc/attention_mma.cu, which a window wider
than everything sends a step to): what is no number, scales that are not positive, many keys, and weights of which the last bits decide."""
import pytest
import torch

from llmgen_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HD, PAGE, WIDE = 128, 16, 1 << 24


def rnd(shape, seed, scale=1.0):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(torch.bfloat16)


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def attend(q, ks, vs, news, window=0, scale=HD ** -0.5):
    """q [tokens, heads, HD] of sequences with keys ks[s], values vs[s] [ctx, kv heads, HD] and news[s] new tokens."""
    T, nq, nkv = q.shape[0], q.shape[1], ks[0].shape[1]
    blocks = [-(-len(k) // PAGE) for k in ks]
    most = max(blocks)
    kc, vc = (torch.zeros(sum(blocks), nkv, PAGE, HD, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    bt, at, tiles, cu = torch.zeros(len(ks), most, dtype=torch.int32), 0, [], [0]
    for s, (k, v, n, m) in enumerate(zip(ks, vs, news, blocks)):
        bt[s, :m] = torch.arange(at, at + m, dtype=torch.int32)
        for cache, x in ((kc, k), (vc, v)):
            padded = torch.zeros(m * PAGE, nkv, HD, dtype=torch.bfloat16)
            padded[:len(x)] = x
            cache[at:at + m] = padded.view(m, PAGE, nkv, HD).transpose(1, 2).to(DEV)
        at += m
        tiles += [(s, q0) for q0 in range(0, n, 64)]
        cu.append(cu[-1] + n)
    out = torch.full((T, nq * HD), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.attention_mma(out, q.reshape(T, nq * HD).to(DEV), kc, vc, bt.to(DEV), most, ints([len(k) for k in ks]), ints(cu), ints([t[0] for t in tiles]),
                      ints([t[1] for t in tiles]), len(tiles), nq, nkv, HD, HD, PAGE, window, scale)
    torch.cuda.synchronize()
    ops.check_tc_errors(out.device)
    return out.view(T, nq, HD)


def plain(q, k, v, scale=HD ** -0.5):
    """One sequence in float64, its last len(q) tokens."""
    n, ctx, group = len(q), len(k), q.shape[1] // k.shape[1]
    k, v = (x.double().repeat_interleave(group, 1) for x in (k, v))
    z = torch.einsum("thd,jhd->htj", q.double(), k) * scale
    z = z.masked_fill((torch.arange(ctx)[None, :] > torch.arange(ctx - n, ctx)[:, None])[None], float("-inf"))
    return torch.einsum("htj,jhd->thd", torch.softmax(z, 2), v)


@pytest.mark.parametrize("scale", [-0.09, 0.0])
def test_a_scale_that_is_not_positive(scale):
    """Scores of up to a hundred either way: against the largest product instead of the largest score the powers would overflow."""
    q, k, v = rnd((200, 4, HD), 1, 24.0), rnd((300, 2, HD), 2), rnd((300, 2, HD), 3)
    got, want = attend(q, [k], [v], [200], scale=scale).cpu().double(), plain(q, k, v, scale)
    # one rounding to bfloat16 (2^-8 of the value at most), and before it float32 sums: 300 terms, scores of 128 products each, as good as 128 2^-24 of the sum of their magnitudes
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + 2.0 ** -24 * (300 + 128 * 0.09 * 4.5 * float(q.double().abs().sum(2).max())) * 4.5).all())


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_what_is_no_number_stays_visible(value):
    q, k, v = rnd((300, 4, HD), 1), rnd((300, 2, HD), 2), rnd((300, 2, HD), 3)
    clean = attend(q, [k], [v], [300])
    bad = q.clone()
    bad[150, 1, 7] = value
    for window in (0, WIDE):
        out = attend(bad, [k], [v], [300], window=window)
        assert bool(torch.isnan(out[150, 1]).all())                      # its own row and head
    out = attend(bad, [k], [v], [300])
    out[150, 1] = clean[150, 1]
    assert torch.equal(out, clean)                                       # and no other
    bad = k.clone()
    bad[100, 0, 7] = float("nan")
    out = attend(q, [bad], [v], [300])
    assert bool(torch.isnan(out[100:, :2]).all())                        # every row that sees the key, in the heads that read it
    out[100:, :2] = clean[100:, :2]
    assert torch.equal(out, clean)


@pytest.mark.parametrize("ctx,sharp", [(512, 1.0), (4096, 1.0), (4096, 4.0), (16384, 4.0)])
def test_many_keys_lose_no_more_than_on_the_other_tensor_path(ctx, sharp):
    """Values that round to another bfloat16 than the float64 result does: no more of them than `mma.sync` gives, whose sums are float32 too."""
    n, nq = 200, 4
    q, k, v = rnd((n, nq, HD), 1, sharp), rnd((ctx, 2, HD), 2), rnd((ctx, 2, HD), 3) + 1
    want = plain(q, k, v).to(torch.bfloat16)
    wrong = [int((attend(q, [k], [v], [n], window=window).cpu() != want).sum()) for window in (0, WIDE)]
    assert wrong[0] <= wrong[1], wrong


def test_the_last_bits_of_a_weight_count():
    """Eight keys, seven of them the row's best (weight 1) and one of weight p = exp(-d): values -t1, -t2, 0, .., 1 with t1 + t2 the two leading bfloat16 terms of p
    leave p - t1 - t2, which weights kept in one or two terms do not have."""
    seqs, nq, nkv = 40, 4, 2
    low = 4 - (torch.arange(seqs * nkv).double().view(seqs, nkv) + 7) * 2.0 ** -6              # the weak key's score: a bfloat16 value (4 - d, d up to 1.4)
    p = torch.exp(low - 4)
    t1 = p.float().to(torch.bfloat16).double()
    t2 = (p - t1).float().to(torch.bfloat16).double()
    ks, vs = [], []
    for s in range(seqs):
        k, v = torch.zeros(8, nkv, HD), rnd((8, nkv, HD), s).float()
        k[:7, :, 0], k[7, :, 0] = 4.0, low[s].float()
        v[:, :, 5] = 0.0
        v[0, :, 5], v[1, :, 5], v[7, :, 5] = -t1[s].float(), -t2[s].float(), 1.0
        assert torch.equal(k.to(torch.bfloat16).float(), k) and torch.equal(v[:2, :, 5].to(torch.bfloat16).float(), v[:2, :, 5])
        ks.append(k.to(torch.bfloat16)), vs.append(v.to(torch.bfloat16))
    q = torch.zeros(seqs * 8, nq, HD)
    q[:, :, 0] = 8.0
    group = nq // nkv
    p, left = (x.repeat_interleave(group, 1) for x in (p, p - t1 - t2))
    # float32: the exponent is a difference of numbers of up to 6 (2^-23 of them each), the power good to 2 units (2^-22), p's own rounding 2^-24; the sums cancel
    # exactly but for it.  Then one rounding to bfloat16 of the result.
    bound = left.abs() * 2.0 ** -8 + p * (2 * 6 * 2.0 ** -24 + 2.0 ** -22 + 2.0 ** -24)
    one, two = (t1 - t1 - t2).repeat_interleave(group, 1), torch.zeros_like(left)
    assert bool(((one - left).abs() > bound).all()) and float(((two - left).abs() > bound).double().mean()) > 0.25      # what fewer terms give is found
    for window in (0, WIDE):
        got = attend(q.to(torch.bfloat16), ks, vs, [8] * seqs, window=window, scale=0.125).cpu().double().view(seqs, 8, nq, HD)[:, 7, :, 5]
        assert bool(((got * (7 + p) - left).abs() <= bound).all()), float(((got * (7 + p) - left).abs() - bound).max())
