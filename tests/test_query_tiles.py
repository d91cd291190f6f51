"""The list of query tiles of a step against one made tile by tile."""
import random

import pytest


def tile_by_tile(q_lens, starts, n_seqs, bound, bq, window, heaviest_first):
    tiles = []
    for s, n in enumerate(q_lens):
        if bound and n == 0:
            continue
        for start in range(0, max(n, 1), bq):
            keys = starts[s] + min(start + bq, max(n, 1))
            tiles.append((min(keys, window + bq) if window else keys, s, start))
    if heaviest_first:
        tiles.sort(key=lambda t: -t[0])
    if bound:
        tiles += [(0, -1, 0)] * (bound // bq + n_seqs - len(tiles))
    return [t[1] for t in tiles], [t[2] for t in tiles]


@pytest.mark.parametrize("bq", [1, 2, 8, 128])
@pytest.mark.parametrize("window", [0, 40])
@pytest.mark.parametrize("heaviest_first", [False, True])
@pytest.mark.parametrize("bounded", [False, True])
def test_as_tile_by_tile(bq, window, heaviest_first, bounded):
    from llmgen_b200.engine.context import StepMetaBuilder
    from llmgen_b200.parts.attention import add_query_tiles
    rng = random.Random(bq + window)
    for lens in [[], [0], [1], [bq], [bq + 1], [0, 5, 0, 2 * bq, 2 * bq], [7] * 9, [rng.randint(0, 300) for _ in range(12)]]:
        starts = [rng.choice([0, 0, 16, 333]) for _ in lens]
        bound = sum(lens) + rng.randint(1, 40) if bounded else 0
        b = StepMetaBuilder(lens, starts, False, 16, bound)
        name = add_query_tiles(b, bq, window, heaviest_first)
        seq, start = tile_by_tile(lens, starts, len(lens), bound, bq, window, heaviest_first)
        assert b.arrays[name + "_seq"].tolist() == seq and b.arrays[name + "_q0"].tolist() == start
