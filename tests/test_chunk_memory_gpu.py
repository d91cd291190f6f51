"""Matrix memories taken in chunks of 64 tokens (csrc/chunk_memory.cuh) against the plain recurrences, token by token in float64: chunks that
are full, one short and one over, sequences that carry a state into a second step, slots that nobody owns, both storage types."""
import pytest
import torch

from tests.plain import derupel_plain, nasozen_plain

pytestmark = pytest.mark.gpu
DT = {"float32": torch.float32, "bfloat16": torch.bfloat16}
DEV = "cuda:0"
SIZES = [(2, 64, 64), (1, 128, 64), (3, 128, 128), (1, 64, 192)]


def rnd(shape, seed, scale=1.0, dtype=torch.float32):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(dtype)


def off(got, want):
    return float((got.double().cpu() - want.double()).norm() / want.double().norm())


def steps():
    """(lengths, cu_q, slots) of two steps of the same three sequences, with an empty sequence without a slot in the list."""
    for lens in ([1, 64, 65], [130, 63, 200]):
        cu = [0, lens[0], lens[0], lens[0] + lens[1], sum(lens)]
        yield lens, torch.tensor(cu, dtype=torch.int32, device=DEV), torch.tensor([2, -1, 0, 3], dtype=torch.int32, device=DEV)


# rows and states are sums of at most 460 float32 terms whose operands carry 2^-24 each; a few dozen of them per chunk in sequence:
# relative errors of 2-norms stay below 32 * 2^-24 = 2e-6
TOL = 2e-6


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("silu", [True, False])
@pytest.mark.parametrize("H,D,E", SIZES)
def test_constant_decay(H, D, E, silu, dtype):
    from llmgen_b200.kernels import ops
    decay = [1.0, 0.97, 0.5][:H]
    state, want_state = torch.zeros(5, H, D, E, device=DEV), {}
    state[1] = 7.0
    for step, (lens, cu, slots) in enumerate(steps()):
        n = sum(lens)
        packed = rnd((n + 3, H * (2 * D + E) + 8), 10 + step, 0.7, DT[dtype])
        need = ops.linear_attention_scratch_floats(n + 3, 4, H, D, E)
        assert need > 0
        out = torch.full((n + 3, H * E), 3.0, device=DEV)
        ops.linear_attention(out, packed.to(DEV), 0, H * D, 2 * H * D, state, torch.tensor(decay, device=DEV), cu, slots, 4, H, D, E, silu=silu,
                             scratch=torch.full((need,), float("nan"), device=DEV))
        at, rows = 0, []
        for i, m in enumerate(lens):
            x = packed[at:at + m].double()
            f = derupel_plain.silu if silu else (lambda z: z)
            q, k, v = f(x[:, :H * D]).view(m, H, D), f(x[:, H * D:2 * H * D]).view(m, H, D), f(x[:, 2 * H * D:2 * H * D + H * E]).view(m, H, E)
            want, want_state[i] = derupel_plain.decayed_outer_product_scan(q, k, v, decay, want_state.get(i))
            rows.append(want.reshape(m, -1))
            at += m
        # (all rows together: a single short row may be what a cancellation left)
        assert off(out[:n], torch.cat(rows)) < TOL
        assert float(out[n:].min()) == 3.0
    for i, slot in enumerate((2, 0, 3)):
        assert off(state[slot], want_state[i]) < TOL
    assert bool((state[1] == 7.0).all()) and float(state[4].abs().sum()) == 0.0


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("forget", [4.0, 0.0, -9.0])
@pytest.mark.parametrize("H,D,E", SIZES)
def test_running_maximum(H, D, E, forget, dtype):
    """`forget`: what the forget gates lie around, from memories that keep hundreds of tokens to ones that drop each at once."""
    from llmgen_b200.kernels import ops
    cap, size = 12.0, H * D * E + H * D + H
    state, st = torch.zeros(5, size, device=DEV), {}
    state[1] = 7.0
    bi, bf = rnd((H,), 1), rnd((H,), 2, 0.2) + forget
    for step, (lens, cu, slots) in enumerate(steps()):
        n = sum(lens)
        packed = rnd((n + 3, H * (2 * D + E) + 2 * H + 8 - 2 * H % 8), 20 + step, 1.0, DT[dtype])
        x = packed.to(DEV)
        q, k, v, gi, gf = (x[:, a:b] for a, b in ((0, H * D), (H * D, 2 * H * D), (2 * H * D, 2 * H * D + H * E), (H * (2 * D + E), H * (2 * D + E) + H),
                                                  (H * (2 * D + E) + H, H * (2 * D + E) + 2 * H)))
        gates = torch.zeros(n + 3, 4 * H, device=DEV)
        ops.mlstm_gates(gates, q, k, gi, gf, bi.to(DEV), bf.to(DEV), state[:, H * D * E + H * D:], cu, slots, 4, H, D, cap, D ** -0.5)
        need = ops.memory_scan_scratch_floats(n + 3, 4, H, D, E, "mlstm")
        assert need > 0
        out = torch.full((n + 3, H * E), 3.0, device=DEV)
        ops.memory_scan(out, q, k, v, None, gates, state, cu, slots, 4, H, D, E, "mlstm", r_scale=D ** -0.5, den_eps=1e-6,
                        scratch=torch.full((need,), float("nan"), device=DEV))
        at = 0
        for i, m in enumerate(lens):
            y = packed[at:at + m].double()
            li = cap * torch.tanh((y[:, H * (2 * D + E):H * (2 * D + E) + H] + bi.double()) / cap)
            lf = torch.nn.functional.logsigmoid(cap * torch.tanh((y[:, H * (2 * D + E) + H:H * (2 * D + E) + 2 * H] + bf.double()) / cap))
            want, st[i] = nasozen_plain.mlstm_memory(y[:, :H * D].view(m, H, D) * D ** -0.5, y[:, H * D:2 * H * D].view(m, H, D),
                                                     y[:, 2 * H * D:2 * H * D + H * E].view(m, H, E), li, lf, st.get(i))
            # (a row whose denominator is what a cancellation left holds fewer digits than the sums it came from)
            assert off(out[at:at + m], want.reshape(m, -1)) < 50 * TOL
            at += m
        assert float(out[n:].min()) == 3.0
    for i, slot in enumerate((2, 0, 3)):
        S, nn, mx = st[i]
        assert off(state[slot, :H * D * E], S.reshape(-1)) < TOL and off(state[slot, H * D * E:H * D * E + H * D], nn.reshape(-1)) < TOL
        assert off(state[slot, H * D * E + H * D:], mx) < TOL
    assert bool((state[1] == 7.0).all())


def test_rows_that_are_no_16_byte_vectors_take_the_walk():
    """The sizes fit, the addresses do not: the same results by the other kernels."""
    from llmgen_b200.kernels import ops
    H, D, E, n = 1, 64, 64, 150
    packed = rnd((n, 3 * 64 + 3), 5, 0.7, torch.bfloat16).to(DEV)[:, 1:]
    cu, slots = torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.tensor([0], dtype=torch.int32, device=DEV)
    state, out = torch.zeros(1, H, D, E, device=DEV), torch.empty(n, E, device=DEV)
    scratch = torch.empty(ops.linear_attention_scratch_floats(n, 1, H, D, E), device=DEV)
    ops.linear_attention(out, packed, 0, 64, 128, state, torch.tensor([0.9], device=DEV), cu, slots, 1, H, D, E, scratch=scratch)
    x = derupel_plain.silu(packed[:, :192].double().cpu()).view(n, 3, 1, 64)
    want, last = derupel_plain.decayed_outer_product_scan(x[:, 0], x[:, 1], x[:, 2], [0.9])
    assert off(out, want.reshape(n, -1)) < TOL and off(state[0], last) < TOL
