"""The memory under a running maximum walked by more blocks than the SMs hold at once (csrc/memory_scan.cu): every tile of columns reads a head's n, one
block writes it."""
import pytest
import torch

from llmgen_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,D,E,seqs", [(2, 64, 64, 200), (4, 64, 128, 150), (1, 32, 24, 700), (16, 128, 128, 9)])
def test_every_tile_reads_n_as_it_was(H, D, E, seqs):
    g = torch.Generator().manual_seed(3)
    rnd = lambda *shape: torch.randn(*shape, generator=g).to(DEV)
    q, k, v, S0, n0, m0 = rnd(seqs, H, D), rnd(seqs, H, D), rnd(seqs, H, E), rnd(seqs, H, D, E), rnd(seqs, H, D), rnd(seqs, H)
    gi, gf, gates = rnd(seqs, H), rnd(seqs, H) + 2, torch.zeros(seqs, H, 4, device=DEV)
    cu, slots, scale = torch.arange(seqs + 1, dtype=torch.int32, device=DEV), torch.arange(seqs, dtype=torch.int32, device=DEV), D ** -0.5
    for turn in range(5):
        state, out = torch.cat([S0.reshape(seqs, -1), n0.reshape(seqs, -1), m0], 1).contiguous(), torch.empty(seqs, H * E, device=DEV)
        ops.mlstm_gates(gates.view(seqs, -1), q.view(seqs, -1), k.view(seqs, -1), gi, gf, None, None, state[:, H * D * (E + 1):], cu, slots, seqs, H, D, 12.0, scale)
        ops.memory_scan(out, q.view(seqs, -1), k.view(seqs, -1), v.view(seqs, -1), None, gates, state, cu, slots, seqs, H, D, E, "mlstm", r_scale=scale, den_eps=1e-6)
        i, f, m = (gates[..., c].double() for c in (0, 1, 3))
        top = torch.maximum(f + m, i)
        keep, take = torch.exp(f + m - top)[..., None], torch.exp(i - top)[..., None]
        S = keep[..., None] * S0.double() + (take * k.double())[..., None] * v.double()[:, :, None]
        n = keep * n0.double() + take * k.double()
        r = q.double() * scale
        num, den = torch.einsum("shde,shd->she", S, r), torch.maximum((n * r).sum(-1).abs(), torch.exp(-top))[..., None] + 1e-6
        # float32 sums of D products: each good to a few 2^-24 of the sum of the magnitudes; the quotient has both
        slack = 64 * 2.0 ** -24 * (torch.einsum("shde,shd->she", S.abs(), r.abs()) + num.abs() * (n * r).abs().sum(-1)[..., None] / den) / den
        assert bool(((out.view(seqs, H, E).double() - num / den).abs() <= slack).all()), turn
        got = state[:, H * D * E:H * D * (E + 1)].view(seqs, H, D).double()
        assert bool(((got - n).abs() <= 8 * 2.0 ** -24 * (keep * n0.double().abs() + take * k.double().abs())).all())
