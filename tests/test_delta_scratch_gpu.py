"""The chunks' scratch of the delta rule with one decay per head: one array an engine, within what is left for it."""
import pytest
import torch

pytestmark = pytest.mark.gpu

H, G, D, E, W = 4, 2, 64, 64, 64


def a_mixer():
    from llmgen_b200.parts.registry import build_mixer, mixer_class
    from llmgen_b200.parts.spec import HeadDecayDeltaSpec, RMSNormSpec, ShortConvSpec
    from llmgen_b200.weights import weights_from_dict
    g = torch.Generator().manual_seed(1)
    w = lambda *shape: (torch.randn(*shape, generator=g) * 0.1).to(torch.bfloat16)
    spec = HeadDecayDeltaSpec(hidden_size=W, num_heads=H, num_kv_heads=G, key_dim=D, value_dim=E, conv=ShortConvSpec(2 * G * D + H * E, 4, "cw"),
                              conv_weights=("cq", "ck", "cv"), q_proj="q", k_proj="k", v_proj="v", beta_proj="b", decay_proj="a", decay_bias="db",
                              decay_log="al", gate_proj="g", o_proj="o", out_norm=RMSNormSpec(E, 1e-5, "n"))
    tensors = {"q": w(G * D, W), "k": w(G * D, W), "v": w(H * E, W), "b": w(H, W), "a": w(H, W), "db": torch.zeros(H), "al": torch.zeros(H),
               "g": w(H * E, W), "o": w(W, H * E), "n": torch.ones(E), "cq": w(G * D, 4).float(), "ck": w(G * D, 4).float(), "cv": w(H * E, 4).float()}
    return build_mixer(spec, weights_from_dict(tensors, mixer_class(spec).weight_decls(spec)), torch.bfloat16, "cuda")


def test_many_single_tokens_beside_a_portion_stay_within_the_reserve():
    from llmgen_b200.kernels import ops
    from llmgen_b200.parts.base import LayerCache
    from tests.util import manual_context
    part, workspace = a_mixer(), None
    for lens in ([256], [512], [30] * 10, [1] * 255 + [257]):
        ctx = manual_context(lens, [0] * len(lens), [[0] * 64] * len(lens), 16, torch.bfloat16, max_step_tokens=512)
        ctx.max_seqs_bound = 256
        workspace = ctx.workspace = workspace or ctx.workspace
        state = torch.zeros(len(lens), *part.state_request().shape, device="cuda")
        part.forward(ctx, torch.randn(sum(lens), W, device="cuda").to(torch.bfloat16), LayerCache(state=state))
    torch.cuda.synchronize()
    assert [k for k in workspace._buffers if "chunks" in k] == ["hdelta_chunks:flat:torch.float32"] and not workspace._retired
    said = part.workspace_bytes(512) + part.sequence_bytes(512, 256)
    # (what is said counts a sliced product's slices, which this step's products do not make)
    assert workspace.bytes_held() <= said < workspace.bytes_held() + ops.SLICED_PRODUCT_BYTES + (1 << 20)


def test_the_engine_leaves_it():
    from types import SimpleNamespace
    from llmgen_b200.engine.executor import Executor
    part = a_mixer()
    layer = SimpleNamespace(mixer=part, workspace_bytes=part.workspace_bytes)
    model = SimpleNamespace(spec=SimpleNamespace(hidden_size=W, vocab_size=100), layers=[layer], mixers=lambda: [part, None])
    reserve = lambda seqs: Executor._activation_reserve(SimpleNamespace(model=model, dtype=torch.bfloat16, limits=SimpleNamespace(max_step_tokens=512,
                                                                                                                                max_num_seqs=seqs)))
    assert reserve(256) - reserve(64) == part.sequence_bytes(512, 256) - part.sequence_bytes(512, 64) + 2 * 192 * 100 * 4
    assert reserve(1000) == reserve(512) + 2 * 488 * 100 * 4
