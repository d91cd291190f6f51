"""The order of the prompt attention's roles (csrc/attention_tc.cu): P V of a tile of keys reads what every softmax warp has
written.  Warps may be a tile apart, so an arrival has to say for which tile it is."""
import os
import re
import tempfile

import pytest
import torch

from tests.util import ROOT, TINY, Driver, logits_close, make_folder, needle_ids, reference


def early_products(n_warps, n_tiles, n_barriers):
    """Every order of the roles, as the kernel's waits allow it: warp w finishes tile t (an arrival on barrier t % n_barriers) once its scores
    are there, those of tile t after P V of tile t - 2; P V of tile j follows the (j // n_barriers)-th completed phase of its barrier.  Returns
    the tiles whose P V can run while a warp has not finished them."""
    found, seen = set(), set()
    todo = [((0,) * n_warps, 0)]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        done, issued = state
        arrived = [sum(1 for n in done for t in range(n) if t % n_barriers == b) for b in range(n_barriers)]
        if issued < n_tiles and arrived[issued % n_barriers] >= (issued // n_barriers + 1) * n_warps:
            if min(done) <= issued:
                found.add(issued)
            todo.append((done, issued + 1))
        for w in range(n_warps):
            if done[w] < n_tiles and (done[w] < 2 or issued >= done[w] - 1):
                todo.append((done[:w] + (done[w] + 1,) + done[w + 1:], issued))
    return found


def test_a_barrier_for_each_of_two_tiles_holds_the_products_back():
    assert early_products(3, 5, 2) == set()
    assert early_products(3, 5, 1) == {0, 1, 2, 3}         # one barrier: a warp that is ahead stands in for one that is behind


def test_the_kernel_waits_and_arrives_by_tile():
    with open(os.path.join(ROOT, "llmgen_b200", "csrc", "attention_tc.cu")) as f:
        src = f.read()
    assert re.findall(r"mbar_(?:wait_warp|arrive)\(tc::smem_u32\(([^()]*p_full[^()]*)\)", src) == ["&p_full[st]"] * 2
    assert "mbar_wait_warp(tc::smem_u32(&p_full[st]), (j >> 1) & 1" in src


@pytest.mark.gpu
def test_freshly_loaded_models_give_the_same_rows():
    """A portion of 129 tokens behind 236, three tiles of keys, as the first steps of a hundred freshly loaded models: then code and
    weights are not in the caches and warps drift apart.  (With one barrier for all tiles up to one load in fourteen gave rows that were
    not the others'.)"""
    with tempfile.TemporaryDirectory() as tmp:
        path = make_folder(tmp, "D", num_hidden_layers=1, layer_types=["full_attention"])
        ids = needle_ids(365, TINY["D"][0]["vocab_size"], 128, 5)
        ref, bound = reference(path, ids)
        first = None
        for _ in range(100):
            d = Driver(path, "bfloat16", 1024, TINY["D"][5], eager=False)
            at = 0
            for n in (57, 129, 50, 129):
                got = d.step([("p", ids[at:at + n], range(n))], end=["p"] if at + n == len(ids) else [])
                at += n
            if first is None:
                first = got
                logits_close(first, ref[236:], "bfloat16", bound)
            assert torch.equal(got, first)
            assert d.executor.status_dev.tolist() == [0, 0]
