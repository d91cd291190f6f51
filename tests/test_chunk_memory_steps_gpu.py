"""Matrix memories in steps of many sequences (csrc/chunk_memory.cuh beside the walks of csrc/linear_attention.cu and csrc/memory_scan.cu): what a
sequence's tokens give follows from its own portion and state, whatever else the step holds."""
import pytest
import torch

from llmgen_b200.kernels import ops

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
DEV = "cuda:0"
H, D, E, CAP = 2, 64, 64, 12.0
SIZE = H * D * E + H * D + H


def rnd(shape, seed, scale=1.0, dtype=torch.float32):
    return (torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale).to(dtype)


def ints(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def offsets(lens):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    return ints(cu)


def linear(x, state, lens, longest=0, scratch=True):
    """One step over rows x [n, H (2 D + E)] of sequences of `lens` tokens, sequence s in state[s]; the outputs."""
    n = len(x)
    out = torch.full((n, H * E), 3.0, device=DEV)
    need = ops.linear_attention_scratch_floats(n, len(lens), H, D, E) if scratch else 0
    ops.linear_attention(out, x, 0, H * D, 2 * H * D, state, torch.tensor([0.97, 0.5], device=DEV), offsets(lens), ints(list(range(len(lens)))), len(lens), H, D, E,
                         scratch=torch.full((need,), float("nan"), device=DEV) if need else None, **({"longest": longest} if longest else {}))
    return out


def mlstm(x, state, lens, longest=0, scratch=True):
    """The same for the memory under a running maximum; the gates' columns follow q, k and v."""
    n, slots = len(x), ints(list(range(len(lens))))
    q, k, v = x[:, :H * D], x[:, H * D:2 * H * D], x[:, 2 * H * D:2 * H * D + H * E]
    gates, at, hint = torch.zeros(n, 4 * H, device=DEV), H * (2 * D + E), {"longest": longest} if longest else {}
    ops.mlstm_gates(gates, q, k, x[:, at:at + H], x[:, at + H:at + 2 * H], None, torch.tensor([3.0, 0.0], device=DEV), state[:, H * D * E + H * D:], offsets(lens),
                    slots, len(lens), H, D, CAP, D ** -0.5, **hint)
    out = torch.full((n, H * E), 3.0, device=DEV)
    need = ops.memory_scan_scratch_floats(n, len(lens), H, D, E, "mlstm") if scratch else 0
    ops.memory_scan(out, q, k, v, None, gates, state, offsets(lens), slots, len(lens), H, D, E, "mlstm", r_scale=D ** -0.5, den_eps=1e-6,
                    scratch=torch.full((need,), float("nan"), device=DEV) if need else None, **hint)
    return out


def fresh(form, n):
    return rnd((n, H, D, E), 1, 0.3).to(DEV) if form is linear else rnd((n, SIZE), 1, 0.3).to(DEV)


def rows(n, dtype, seed=2):
    return rnd((n, H * (2 * D + E) + 8), seed, 0.7, DT[dtype]).to(DEV)


LENS = [1] * 150
for at, n in ((0, 130), (30, 32), (37, 64), (40, 65), (70, 48), (71, 49), (100, 0), (131, 300), (149, 200)):
    LENS[at] = n


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("form", [linear, mlstm])
def test_a_sequence_gives_what_it_gives_alone(form, dtype):
    x, state = rows(sum(LENS), dtype), fresh(form, len(LENS))
    before = state.clone()
    out = form(x, state, LENS)
    at = 0
    for s, n in enumerate(LENS):
        if s in (0, 1, 30, 37, 40, 70, 71, 72, 131, 148, 149):
            own = before[s:s + 1].clone()
            assert torch.equal(form(x[at:at + n], own, [n]), out[at:at + n]), (s, n)
            assert torch.equal(own, state[s:s + 1]), (s, n)
        at += n
    assert torch.equal(state[100], before[100])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("form", [linear, mlstm])
def test_a_sequence_among_more_chunks_than_the_sms_take_at_once(form, dtype):
    """60 sequences of 100 tokens and 2 heads: 240 blocks of outputs, two an SM; alone a sequence's blocks have an SM each."""
    lens = [100] * 60
    x, state = rows(sum(lens), dtype), fresh(form, len(lens))
    before = state.clone()
    out = form(x, state, lens)
    for s in (0, 31, 59):
        alone = before[s:s + 1].clone()
        assert torch.equal(form(x[100 * s:100 * (s + 1)].contiguous(), alone, [100]), out[100 * s:100 * (s + 1)])
        assert torch.equal(alone, state[s:s + 1])


@pytest.mark.parametrize("form", [linear, mlstm])
def test_scratch_follows_what_long_sequences_can_be_there(form):
    entries = D * E + (D if form is mlstm else 0)
    need = ops.memory_scan_scratch_floats if form is mlstm else ops.linear_attention_scratch_floats
    last = ("mlstm",) if form is mlstm else ()
    few = need(256, 8, H, D, E, *last)
    # 256 tokens are at most four whole chunks and the shorter chunks of five sequences of more than 48 tokens
    assert 0 < few <= need(256, 256, H, D, E, *last) <= 9 * H * (entries + 2) + 256 * H


@pytest.mark.parametrize("form", [linear, mlstm])
def test_single_tokens_are_walked_without_scratch(form):
    x, lens = rows(200, "bfloat16"), [1] * 200
    a, b = fresh(form, 200), fresh(form, 200)
    assert torch.equal(form(x, a, lens, longest=1, scratch=False), form(x, b, lens)) and torch.equal(a, b)


def launched(f):
    before = ops.launches()
    f()
    return ops.launches() - before


@pytest.mark.parametrize("n", [65, 100, 256])
def test_linear_attention_of_up_to_256_tokens_needs_no_scratch(n):
    x, want_state, state = rows(n, "bfloat16"), fresh(linear, 1), fresh(linear, 1)
    want, out = linear(x, want_state, [n]), linear(x, state, [n], scratch=False)
    # (float32 sums of at most 256 terms of the same size in another order)
    assert float((out - want).norm() / want.norm()) < 2e-6 and float((state - want_state).norm() / want_state.norm()) < 2e-6


def test_a_step_that_needs_scratch_for_its_segments_says_so():
    x, state = rows(257, "bfloat16"), fresh(linear, 1)
    with pytest.raises(ops.KernelError, match="scratch"):
        linear(x, state, [257], scratch=False)


def test_launches_are_counted_as_they_happen():
    x, wide = rows(200, "bfloat16"), rows(200, "bfloat16")[:, 1:]        # (the second's rows start off 16-byte boundaries)
    assert launched(lambda: linear(x, fresh(linear, 1), [200])) == 4
    assert launched(lambda: linear(wide, fresh(linear, 1), [200])) == 1
    assert launched(lambda: linear(x, fresh(linear, 1), [200], scratch=False)) == 1
    assert launched(lambda: linear(x, fresh(linear, 200), [1] * 200, longest=1)) == 1
    assert launched(lambda: mlstm(x, fresh(mlstm, 1), [200])) == 2 + 4
    assert launched(lambda: mlstm(wide, fresh(mlstm, 1), [200])) == 2 + 1


def a_mixer(form):
    """(the part, the state's shape) of one layer around the memory."""
    from llmgen_b200.parts.registry import build_mixer, mixer_class
    from llmgen_b200.parts.spec import LinearAttentionSpec, MLSTMSpec
    from llmgen_b200.weights import weights_from_dict
    W, w = 64, lambda i, rows, cols: rnd((rows, cols), i, 0.1, torch.bfloat16)
    if form is linear:
        spec = LinearAttentionSpec(hidden_size=W, num_heads=H, key_dim=D, value_dim=E, decay=(0.9, 0.5), q_proj="q", k_proj="k", v_proj="v", o_proj="o")
        tensors, shape = {}, (H, D, E)
    else:
        spec = MLSTMSpec(hidden_size=W, num_heads=H, key_dim=D, value_dim=E, gate_cap=CAP, eps=1e-5, q_proj="q", k_proj="k", v_proj="v", i_proj="i", f_proj="f",
                         gate_proj="g", o_proj="o", out_gain="n", den_eps=1e-6)
        tensors, shape = {"i": w(5, H, W), "f": w(6, H, W), "g": w(7, H * E, W), "n": torch.ones(H * E)}, (SIZE,)
    tensors.update({"q": w(1, H * D, W), "k": w(2, H * D, W), "v": w(3, H * E, W), "o": w(4, W, H * E)})
    return build_mixer(spec, weights_from_dict(tensors, mixer_class(spec).weight_decls(spec)), torch.bfloat16, DEV), shape


@pytest.mark.parametrize("form", [linear, mlstm])
def test_a_workspace_keeps_one_array_for_the_chunks(form):
    """Steps of rising sizes, as when graphs are captured: no array is outgrown, and what is held is what was said to be."""
    from llmgen_b200.parts.base import LayerCache
    from tests.util import manual_context
    part, shape = a_mixer(form)
    workspace = None
    for lens in ([1] * 80, [1] * 256, [100], [60] * 3, [500], [300, 1, 1], [70] * 14, [1024]):
        ctx = manual_context(lens, [0] * len(lens), [[0] * 64] * len(lens), 16, torch.bfloat16, max_step_tokens=1024)
        ctx.max_seqs_bound = 256
        workspace = ctx.workspace = workspace or ctx.workspace
        part.forward(ctx, rnd((sum(lens), 64), 9, 1.0, torch.bfloat16).to(DEV), LayerCache(state=torch.zeros(len(lens), *shape, device=DEV)))
    torch.cuda.synchronize()
    held = [b for name, b in workspace._buffers.items() if "chunks" in name]
    assert len(held) == 1 and all(b.numel() < 4096 for b in workspace._retired)
    assert held[0].numel() * 4 <= part.workspace_bytes(1024) and workspace.bytes_held() <= part.workspace_bytes(1024) + ops.SLICED_PRODUCT_BYTES + (1 << 20)


def same(a, b):
    return torch.allclose(a, b, rtol=0, atol=0, equal_nan=True)


# what a value of `where` (head 1, sequence 1) is made, at which of its 200 tokens
ODD = [("v", float("inf"), 70), ("v", float("nan"), 127), ("k", float("-inf"), 10), ("k", float("nan"), 199), ("q", float("inf"), 64), ("q", float("nan"), 130),
       ("v", 2.9e38, 100), ("state", float("inf"), -1), ("state", float("nan"), -1), ("n", float("inf"), -1), ("f", float("-inf"), 90), ("f", -3e6, 30), ("i", float("-inf"), 77), ("f", float("nan"), 150)]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("form", [linear, mlstm])
@pytest.mark.parametrize("where,value,token", ODD)
def test_what_is_no_ordinary_number_goes_the_way_of_the_walk(where, value, token, form, dtype, monkeypatch):
    """Infinities, NaN, values beyond what bfloat16 terms hold, gates that close at once: the sequence's head gives what the walk token by token
    gives, from its own token on and not before, and nothing else changes."""
    if form is linear and where in ("n", "f", "i"):
        pytest.skip("gates and n belong to the running maximum")
    lens = [100, 200, 30, 130]
    x, state = rows(sum(lens), dtype), fresh(form, len(lens))
    clean_state = state.clone()
    clean = form(x, clean_state, lens)
    x = x.clone()
    if where in ("q", "k", "v"):
        x[100 + token, {"q": 0, "k": H * D, "v": 2 * H * D}[where] + D + 5] = value
    elif where == "state":
        state.view(len(lens), -1)[1, D * E + 3 * E + 7] = value
    elif where == "n":
        state[1, H * D * E + D + 4] = value
    elif where in ("f", "i"):
        def gates_with(gates, *args, _inner=ops.mlstm_gates, **kwargs):
            _inner(gates, *args, **kwargs)
            row = (100 if len(gates) == sum(lens) else 0) + token
            gates.view(len(gates), H, 4)[row, 1, 1 if where == "f" else 0] = value
        monkeypatch.setattr(ops, "mlstm_gates", gates_with)
    alone = state[1:2].clone()
    out, walk = form(x, state, lens), form(x[100:300], alone, [200], scratch=False)
    at = slice(E, 2 * E)
    assert same(out[100:300, at], walk[:, at])
    entries = torch.zeros(SIZE if form is mlstm else H * D * E, dtype=torch.bool, device=DEV)
    entries[D * E:2 * D * E] = True
    if form is mlstm:
        entries[H * D * E + D:H * D * E + 2 * D] = True
        entries[H * D * E + H * D:] = state.view(len(lens), -1)[1, H * D * E + H * D:] == alone[0, H * D * E + H * D:]      # (m is the gates' kernel's)
    assert same(state.view(len(lens), -1)[1][entries], alone.view(-1)[entries])
    assert bool(torch.isfinite(out[100:100 + max(token, 0), at]).all()) and (where not in ("q", "k", "v") or abs(value) < 1e39 or not bool(torch.isfinite(out[100 + token, at]).all()))
    out[100:300, at] = clean[100:300, at]
    assert same(out, clean)
    others = ~entries if form is linear else ~entries & (torch.arange(SIZE, device=DEV) < H * D * E + H * D)
    assert same(state.view(len(lens), -1)[1][others], clean_state.view(len(lens), -1)[1][others])
    assert same(state[[0, 2, 3]], clean_state[[0, 2, 3]])
