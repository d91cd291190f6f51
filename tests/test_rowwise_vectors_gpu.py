"""Row-wise kernels that take whole vectors where sizes and addresses allow it: rows of one vector, of a warp's and a block's edge, of the widest
block, and just beyond, against float64.  float32 arithmetic on the stored values: 2e-6 relative to the largest value (sums of up to 4,100
squares and an exponential), and the storage type's own rounding (2^-8) on top where that is bfloat16."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
DEV = "cuda:0"
WIDTHS = [4, 12, 128, 132, 260, 1030, 2048, 4096, 4100]


def rnd(shape, seed, scale=1.0, dtype=torch.float32):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(dtype)


def close(got, want, tol):
    err = float((got.double().cpu() - want).abs().max() / want.abs().max())
    assert err < tol, err


def tol(dtype):
    return 2e-6 if dtype == "float32" else 2.0 ** -8


def norm(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H", WIDTHS)
@pytest.mark.parametrize("pair,chained,sliced", [(False, False, False), (True, False, True), (False, True, True), (True, True, False)])
def test_norm_add(H, pair, chained, sliced, dtype):
    from llmgen_b200.kernels import ops
    from llmgen_b200.kernels.ops import Partials
    n, dt, eps = 5, DT[dtype], 1e-6
    resid, w, w2 = rnd((n, H), 1, 2.0), 1 + rnd((H,), 2, 0.2), 1 + rnd((H,), 3, 0.2)
    first = rnd((3, n, H), 4, 0.5) if sliced else rnd((n, H), 4, 0.5, dt)
    other = rnd((n, H), 5, 0.5, dt)
    a64 = first.double().sum(0) if sliced else first.double()
    want = resid.double() + norm(0.7 * a64 + 0.3 * other.double() if pair else a64, w.double(), eps)
    r, copy = resid.to(DEV), torch.empty(n, H, dtype=dt, device=DEV)
    y = Partials(first.to(DEV)) if sliced else first.to(DEV)
    if pair:
        y = ops.WeightedPair(y, 0.7, other.to(DEV), 0.3)
    ops.norm_add(r, y, w.to(DEV), eps, copy, dt, next_gain=w2.to(DEV) if chained else None, next_eps=eps)
    close(r, want, 2e-6)
    close(copy, norm(want, w2.double(), eps) if chained else want, tol(dtype))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H", WIDTHS)
@pytest.mark.parametrize("heads,gate_form,offset", [(1, "sigmoid", 8), (3, "silu", 0), (3, "plain", 4), (2, "silu", 1)])
def test_gated_rmsnorm(H, heads, gate_form, offset, dtype):
    """`offset`: columns before the gate's, which decide whether its rows are whole vectors."""
    from llmgen_b200.kernels import ops
    n, dt, eps = 9, DT[dtype], 1e-6
    o, w = rnd((n * heads, H), 1, 2.0), 1 + rnd((heads, H), 2, 0.2)
    gate = rnd((n, heads * H + 8), 3, 1.0, dt)
    forms = {"sigmoid": torch.sigmoid, "silu": torch.nn.functional.silu, "plain": lambda z: z}
    g64 = forms[gate_form](gate[:, offset:offset + heads * H].double()).reshape(n * heads, H)
    want = norm(o.double(), w.double().repeat(n, 1), eps) * g64
    out = torch.empty(n * heads, H, dtype=dt, device=DEV)
    ops.gated_rmsnorm(out, o.to(DEV), gate.to(DEV)[:, offset:offset + heads * H], w.to(DEV), eps, gate_form=gate_form, heads=heads, gains_per_head=True)
    close(out, want, tol(dtype))


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("F,extra", [(8, 0), (40, 0), (41, 0), (2048, 8), (2048, 3)])
def test_activations(F, extra, dtype):
    from llmgen_b200.kernels import ops
    x = rnd((7, F + extra), 1, 1.5, DT[dtype])
    for name, f in (("relu2", lambda z: torch.relu(z) ** 2), ("tanh", torch.tanh), ("gelu_tanh", lambda z: torch.nn.functional.gelu(z, approximate="tanh"))):
        out = torch.empty(7, F, dtype=DT[dtype], device=DEV)
        ops.act_rows(out, x.to(DEV)[:, :F], name)
        close(out, f(x[:, :F].double()), tol(dtype))


@pytest.mark.parametrize("H", [4, 6, 2048])
def test_casts_and_streams(H):
    from llmgen_b200.kernels import ops
    row, streams = rnd((9, H), 1), torch.empty(9, 3, H, device=DEV)
    ops.stream_spread(streams, row.to(DEV))
    assert all(torch.equal(streams[:, s].cpu(), row) for s in range(3))
    x, back = rnd((9, 3, H), 2), torch.empty(9, H, device=DEV)
    ops.stream_spread(x.to(DEV), back, collapse=True)
    assert torch.equal(back.cpu(), x[:, 0] + x[:, 1] + x[:, 2])
    for dtype in DT.values():
        out = torch.empty(9, H, dtype=dtype, device=DEV)
        ops.cast_rows(out, row.to(DEV))
        assert torch.equal(out.cpu(), row.to(dtype))
