"""Steps of a decoder that routes: a router turns another rounding into another expert, so products of a few tokens keep the sums
that the uncut product has."""
import pytest
import torch

import lulisun_models
import plain_lulisun
from conftest import random_tokens

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


@pytest.mark.parametrize("width, heads", [(1024, 8), (512, 4)])
def test_routed_steps_away_from_near_ties(width, heads, monkeypatch, tmp_path):
    """A decode step whose products are as large as served ones, routers undisturbed, against 64 bits: compared are the sequences
    in which no token's choice, of groups or of experts, hangs on bfloat16's rounding of the router's input."""
    layer = lulisun_models._layer(heads=heads, kv=2, dim=128, vdim=128, scale=0.088, chunk=16, base=10000.0, rot=64, rh=4, rdim=64, rvdim=64,
                                  ls=0.7, rs=0.7, mlp=lulisun_models._moe(16, 2, 128, groups=(4, 2), shared=256))
    cfg = {"architecture": "Lulisun", "vocab": 300, "width": width, "norm": {"eps": 1e-5}, "layers": [layer] * 2}
    model = lulisun_models.make(tmp_path, f"w{width}", cfg=cfg)
    margins, route = [], plain_lulisun.route

    def recorded(h, w, pre, *, experts, top, groups, keep):
        ids, weights, s = route(h, w, pre, experts=experts, top=top, groups=groups, keep=keep)
        choice = (s + w[pre + "correction"]).view(len(h), groups, -1)
        of_groups = choice.topk(2, -1).values.sum(-1).sort(-1, descending=True)
        kept = torch.zeros(len(h), groups, dtype=torch.bool).scatter_(1, of_groups.indices[:, :keep], True)
        best = choice.masked_fill(~kept[..., None], -9.0).view(len(h), -1).sort(-1, descending=True).values
        margins.append(torch.minimum(of_groups.values[:, keep - 1] - of_groups.values[:, keep], best[:, top - 1] - best[:, top]))
        return ids, weights, s

    monkeypatch.setattr(plain_lulisun, "route", recorded)
    n = 32
    prompts = [random_tokens(3 + i % 5, 300, 100 + i) for i in range(n)]
    want, decided = [], []
    for p in prompts:
        margins.clear()
        want.append(model.plain_logits(p)[-1])
        # a rounding to bfloat16 moves a router's score, a sigmoid of a sum of N(0, 1) terms, by about 2e-3
        decided.append(min(float(m.min()) for m in margins) > 1e-2)
    assert sum(decided) >= n // 4
    from rust_inference_b200.engine.engine import Engine
    eng = Engine.from_pretrained(model.folder, dtype="bfloat16", max_tokens=n * 64, n_slots=n)
    for i in range(0, n, 8):
        slots = [eng.alloc_slot() for _ in range(8)]
        eng.step(slots, [p[:-1] for p in prompts[i:i + 8]], "none")
        got = eng.step(slots, [p[-1:] for p in prompts[i:i + 8]], "last").double().cpu()
        for j in range(8):
            if decided[i + j]:
                w = want[i + j]
                # eight roundings to bfloat16 (2^-9) a layer one after the other; a wrong expert costs 0.1 and more
                assert float((got[j] - w).norm() / w.norm()) <= 2e-2
    eng.check_device_status()
