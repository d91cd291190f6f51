"""Steps of an engine whose latent attention runs on tcgen05 (ranks 256 and 512, a rotated part of 64): portions, and single tokens deep
into their context beside them."""
import pytest
import torch

from tests import derupel_util as du

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eager", [True, False])
@pytest.mark.parametrize("heads,rank", [(8, 256), (16, 512), (5, 256)])
def test_single_tokens_beside_portions(heads, rank, eager):
    layer = du.latent(heads, 16, 64, 24, 40, rank, 0.15, 1000.0, du.dense(80))
    cfg = du.config([layer, layer])
    model, tensors = du.build(cfg, seed=7, dtype="bfloat16")
    drv = du.driver(model, "bfloat16", pool_tokens=640, eager=eager)
    assert model.layers[0].mixer.tc_tile_queries(drv.executor.limits.page_size) == 128 // heads
    ids = {"a": du.ids_for(cfg, 330, 21), "b": du.ids_for(cfg, 180, 22)}
    want = {r: du.plain_logits(cfg, tensors, t) for r, t in ids.items()}
    pos, got = {"a": 0, "b": 0}, {"a": [], "b": []}
    # tokens of a and of b per step: a long portion, single tokens beside portions, both alone, single tokens of both
    for na, nb in ((260, 0), (1, 120), (1, 17), (40, 1), (1, 1), (0, 30), (27, 11)):
        entries, end = [], []
        for r, n in (("a", na), ("b", nb)):
            if n:
                entries.append((r, ids[r][pos[r]:pos[r] + n], list(range(n))))
                pos[r] += n
                end += [r] if pos[r] == len(ids[r]) else []
        out, at = drv.step(entries, end=end), 0
        for r, tokens, _ in entries:
            got[r].append(out[at:at + len(tokens)])
            at += len(tokens)
    for r in ids:
        assert pos[r] == len(ids[r])
        du.assert_close(torch.cat(got[r]), want[r], "bfloat16", r)
