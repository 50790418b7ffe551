"""Steps of a decoder that routes: a router turns another rounding into another expert, so products of a few tokens keep the sums
that the uncut product has."""
import pytest
import torch

import lulisun_models

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _engine(config):
    from rust_inference_b200 import Engine, config_from_dict
    return Engine.from_random(config_from_dict(config), max_tokens=1024, n_slots=4)


def test_the_steps_of_a_routed_decoder_are_marked():
    dense = {"architectures": ["Qwen2ForCausalLM"], "hidden_size": 128, "num_hidden_layers": 1, "num_attention_heads": 2,
             "num_key_value_heads": 1, "head_dim": 64, "intermediate_size": 176, "vocab_size": 264, "rope_theta": 1e6,
             "rms_norm_eps": 1e-6, "attention_bias": True, "tie_word_embeddings": False, "max_position_embeddings": 512}
    for config, routed in ((lulisun_models.CONFIGS["A"], True), (dense, False)):
        eng = _engine(config)
        assert eng.model.routed == routed
        slot = eng.alloc_slot()
        assert eng.make_context([slot], [[1, 2, 3]], [[2]]).routed == routed
        eng.step([slot], [[1, 2, 3]], "last")
        eng.step([slot], [[4]], "last")
        assert eng.decode_graph(1).ctx.routed == routed


@pytest.mark.parametrize("m", [1, 5, 16])
def test_products_of_a_routed_step_keep_their_sums(m):
    from types import SimpleNamespace
    from rust_inference_b200.kernels import linear, ops, tcgen05
    n, k = 2048, 2048
    x = torch.randn(m, k, device=DEV).bfloat16()
    w, w2 = (linear.Weight((torch.randn(n, k, device=DEV) / k ** 0.5).bfloat16()) for _ in range(2))
    assert tcgen05.plan(m, n, k, ops.EPI_STORE_F32)[1] > 1 and tcgen05.plan(m, n, k, ops.EPI_SILU_MUL)[1] > 1
    ctx = SimpleNamespace(routed=True)
    f32 = lambda: torch.full((m, n), 9.0, device=DEV)
    b16 = lambda: f32().bfloat16()
    cols = torch.tensor([700.0], device=DEV)
    pairs = [(linear.logits(x, w, f32(), ctx), tcgen05.gemm(x, w, f32(), ops.EPI_STORE_F32, split_k=1)),
             (linear.logits(x, w, f32(), ctx, silu_cols=cols), tcgen05.gemm(x, w, f32(), ops.EPI_SILU_F32, split_k=1, silu_cols=cols)),
             (linear.project(x, w, b16(), ctx), tcgen05.gemm(x, w, b16(), ops.EPI_STORE, split_k=1)),
             (linear.gated(x, w, w2, b16(), ctx), tcgen05.gemm(x, w, b16(), ops.EPI_SILU_MUL, w2=w2, split_k=1))]
    assert all(torch.equal(got, want) for got, want in pairs)
    ctx.routed = False
    assert not torch.equal(linear.logits(x, w, f32(), ctx), pairs[0][1])          # (cut, the sums are others)
