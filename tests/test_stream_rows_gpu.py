"""The first and the last rewriting of the residual streams: one row in place of equal streams, the sum in place of new ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# vectors of four and single values, one to sixteen streams
@pytest.mark.parametrize("S,H", [(1, 64), (4, 2048), (4, 1028), (3, 37), (8, 4096), (16, 130)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_same_bits_as_with_streams_in_memory(S, H, dtype):
    from llmgen_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(S * H)
    n = 5
    rnd = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    row, mix, out, read, gain, y = rnd(n, H), rnd(S, S), rnd(S), rnd(S), rnd(H), rnd(n, H).to(dtype)

    def spread():
        streams = torch.empty(n, S, H, device="cuda")
        ops.stream_spread(streams, row)
        return streams

    for written in (True, False):
        want_streams, want = spread(), torch.zeros(n, H, dtype=dtype, device="cuda")
        how = (y, mix, out) if written else (None, None, None)
        ops.stream_step(want_streams, *how, read, gain, 1e-5, want, dtype)
        streams, got = torch.full((n, S, H), 7.0, device="cuda"), torch.zeros_like(want)
        ops.stream_step(streams, *how, read, gain, 1e-5, got, dtype, all_equal=row)
        assert torch.equal(got, want)
        assert torch.equal(streams, want_streams) if written else bool((streams == 7.0).all())
    # the last step: the sum of the new streams, and no streams; the row may be the one that was read
    streams, total = rnd(n, S, H), torch.zeros(n, H, device="cuda")
    rewritten, want = streams.clone(), torch.zeros(n, H, device="cuda")
    ops.stream_step(rewritten, y, mix, out, None, None, 0.0, None, dtype)
    ops.stream_spread(rewritten, want, collapse=True)
    kept = streams.clone()
    ops.stream_step(streams, y, mix, out, None, None, 0.0, None, dtype, total=total)
    assert torch.equal(total, want) and torch.equal(streams, kept)
    rewritten = spread()
    ops.stream_step(rewritten, y, mix, out, None, None, 0.0, None, dtype)
    ops.stream_spread(rewritten, want, collapse=True)
    both = row.clone()
    ops.stream_step(streams, y, mix, out, None, None, 0.0, None, dtype, all_equal=both, total=both)
    assert torch.equal(both, want)
    with pytest.raises(ops.KernelError, match="sum"):
        ops.stream_step(streams, None, None, None, read, gain, 1e-5, torch.zeros(n, H, dtype=dtype, device="cuda"), dtype, total=total)
