"""Into how many parts single tokens' keys are cut (`GQAAttention._split`)."""
from types import SimpleNamespace

import pytest

from llmgen_b200.parts.attention import GQAAttention


def parts(nq, nkv, seqs, keys, least, window=0, fixed=True):
    part = SimpleNamespace(nq=nq, nkv=nkv, window=window, chunk=0, sm_count=148)
    ctx = SimpleNamespace(pure_decode=True, n_seqs=seqs, fixed_shapes=fixed, max_ctx_bound=keys, max_ctx=keys)
    return GQAAttention._split(part, ctx, least=least)[0]


@pytest.mark.parametrize("nq,nkv", [(16, 8), (32, 4), (8, 1), (64, 2)])
@pytest.mark.parametrize("seqs", [1, 2, 4, 8, 16, 64])
@pytest.mark.parametrize("keys", [100, 512, 1024, 4096, 40960])
def test_parts_of_128_keys_and_shorter_ones(nq, nkv, seqs, keys):
    blocks = seqs * nkv * -(-(nq // nkv) // 16)
    by_sms = -(-2 * 148 // blocks)
    coarse = max(1, min(by_sms, keys // 128, 64))
    assert parts(nq, nkv, seqs, keys, 128) == coarse                       # a cluster's blocks
    for least in (32, 64):
        n = parts(nq, nkv, seqs, keys, least)
        assert n == coarse or (n >= 2 * coarse and n & (n - 1) == 0 and n <= min(by_sms, keys // least, 64))
        if min(by_sms, keys // least, 64) >= 4 * coarse:
            assert n >= 2 * coarse


def test_a_window_counts_the_keys_that_are_seen():
    assert parts(16, 8, 1, 40960, 32, window=256) == parts(16, 8, 1, 256, 32)


def test_other_steps_are_not_cut():
    part = SimpleNamespace(nq=16, nkv=8, window=0, chunk=0, sm_count=148)
    assert GQAAttention._split(part, SimpleNamespace(pure_decode=False))[0] == 1
