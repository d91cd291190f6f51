"""The few-rows product of a W with few rows: slices of K added up in a cluster, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# clusters of two to eight slices (8, 8, 2, 8, 3, 2, then 4, 5, 6, 7), a last one shorter than the others, tails in N and M, one tile of W
@pytest.mark.parametrize("N,K", [(2048, 2048), (2048, 4096), (1000, 520), (130, 3072), (8, 776), (9000, 512), (4700, 1024), (3712, 1280), (3000, 1536),
                                 (2600, 1792)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_rows_and_their_independence(N, K, out_dtype):
    from llmgen_b200.kernels import ops
    g = torch.Generator().manual_seed(N + K)
    a = torch.randn(64, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=g) * 0.5).to(torch.bfloat16)
    a[63, K - 1] = w[N - 1, K - 1] = 8.0
    ad, wd = a.cuda(), w.cuda()
    ref = a.double() @ w.double().t()
    full = torch.full((65, N + 8), 7.0, dtype=out_dtype, device="cuda")
    ops.gemm_skinny(full[:64, :N], ad, wd)
    torch.cuda.synchronize()
    ops.check_tc_errors(full.device)
    # float32 sums of K products, in slices; a bfloat16 result is rounded once (up to 2^-8 of it)
    assert float((full[:64, :N].double().cpu() - ref).abs().max()) < (2e-5 if out_dtype == torch.float32 else 4e-3) * float(ref.abs().max())
    assert bool((full[64] == 7.0).all()) and bool((full[:, N:] == 7.0).all())
    for rows in (slice(0, 1), slice(5, 8), slice(11, 28), slice(40, 64)):        # a row's sum does not depend on how many there are
        part = torch.empty(rows.stop - rows.start, N, dtype=out_dtype, device="cuda")
        ops.gemm_skinny(part, ad[rows].contiguous(), wd)
        assert torch.equal(part, full[rows, :N])
