"""Which decode steps form their heads inside the attention, and that the step comes out as the separate kernels' does."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
WIDTH = 2048

FORMS = {
    "plain": {}, "biased": dict(qkv_bias=True), "windowed": dict(window=70), "chunked": dict(chunk=64),
    "normed": dict(qk_norm_eps=1e-5), "normed, partly turned": dict(qk_norm_eps=1e-5, rot_dims=64),
    "partly turned": dict(rot_dims=64), "scaled": dict(out_scale=0.7), "values from keys": dict(values_from_keys=True, qk_norm_eps=1e-5),
    "partly turned, scaled, chunked": dict(rot_dims=64, out_scale=0.7, chunk=64),
}
# the separate kernels form these heads from the same float32 sums with the same roundings: the same bits, and they stay in a decoder
# that routes; the others' norms are added up in another order, they come from rows rounded to bfloat16 or are scaled after a rounding
SAME_BITS = {"plain", "biased", "windowed", "chunked"}
SEPARATE = {"gated": dict(out_gate=True), "a gate per head": dict(head_gate=True), "capped": dict(softcap=30.0), "sink": dict(sink=True),
            "another layer's cache": dict(own_kv=False), "a window and a chunk": dict(window=70, chunk=64),
            "values of another size": dict(v_head_dim=64), "odd rotation": dict(rot_dims=36)}


def _layer(form, seed=0, kind="rope"):
    from rust_inference_b200.parts.registry import lookup
    from rust_inference_b200.parts.spec import PartSpec
    form = dict(form)
    rot = form.pop("rot_dims", 128)
    part = lookup("mixer", "gqa_attention")(
        n_heads=8, n_kv_heads=2, head_dim=128, qkv_bias=form.pop("qkv_bias", False),
        position=PartSpec(kind, {"head_dim": 128, "base": 10000.0, "rot_dims": rot}), hidden_size=WIDTH, dtype=torch.bfloat16, device=DEV,
        **form)
    g = torch.Generator(device=DEV).manual_seed(seed)
    part.set_tensors({name: torch.randn(ts.shape, device=DEV, generator=g) * 0.1 + (1.0 if "norm" in name else 0.0) if ts.role == "vector"
                      else (torch.randn(ts.shape, device=DEV, generator=g) / ts.shape[-1] ** 0.5).bfloat16()
                      for name, ts in part.tensor_specs().items()})
    part.prepare(512)
    return part


def _off(t, floats):
    """t's numbers in memory that begins `floats` numbers behind a boundary."""
    room = torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)
    view = room[floats:floats + t.numel()].view(t.shape)
    view.copy_(t)
    return view


def _step(part, monkeypatch, *, separate, routed=False, writes_cache=True, shift=0):
    """One decode step of sequences that end before, at and behind a page's edge: (times the attention formed the heads, its
    result, the cache's keys and values).  shift: the angle tables lie so many floats off a 16-byte boundary."""
    from test_vadodra_gpu import make_ctx
    from rust_inference_b200.cache.sequence_cache import SequenceCache
    from rust_inference_b200.engine.context import Workspace
    from rust_inference_b200.kernels import attention, linear, ops
    cache = SequenceCache([part.cache_request()], max_tokens=2048, max_seq_len=512, dtype=torch.bfloat16, device=DEV, n_slots=6)
    starts = [0, 62, 63, 64, 200]
    slots = [cache.alloc_slot() for _ in starts]
    g = torch.Generator(device=DEV).manual_seed(1)
    layer = cache.layer(0)
    for t in (layer.k, layer.v):
        t.copy_(torch.randn(t.shape, device=DEV, generator=g))
    ctx = make_ctx(cache, slots, starts, [1] * len(starts), torch.bfloat16, Workspace(DEV))
    ctx.routed = routed
    x = torch.randn(len(starts), WIDTH, device=DEV, generator=g).bfloat16()
    residual = torch.zeros(len(starts), WIDTH, device=DEV)
    if shift:
        part.position.cos, part.position.sin = (_off(t, shift) for t in (part.position.cos, part.position.sin))
    runs = []
    with monkeypatch.context() as m:
        # sums in one order, whichever pieces of K arrive first
        m.setattr(linear, "accumulate_split", lambda x, w, acc, ctx: acc.copy_(x.float() @ w.t.float().t()))
        real = attention.FormedHeads.run
        m.setattr(attention.FormedHeads, "run", lambda self, *a, **k: (runs.append(1), real(self, *a, **k))[1])
        if separate:
            m.setattr(attention, "formed_heads", lambda *a, **k: None)
        part.forward(x, residual, ctx, layer, writes_cache)
    torch.cuda.synchronize()
    return len(runs), ctx.buffer("attn_out", (len(starts), part.o_dim), torch.bfloat16).clone(), layer.k.clone(), layer.v.clone()


@pytest.mark.parametrize("name", FORMS)
def test_heads_are_formed_in_the_attention(name, monkeypatch):
    part = _layer(FORMS[name])
    formed, out, k, v = _step(part, monkeypatch, separate=False)
    other, want, k2, v2 = _step(part, monkeypatch, separate=True)
    assert (formed, other) == (1, 0)
    if name in SAME_BITS:
        assert torch.equal(k, k2) and torch.equal(v, v2) and torch.equal(out, want)
    else:
        # one rounding to bfloat16 (2^-8 of a step) more or less in every head and in the result
        for a, b in ((k, k2), (v, v2), (out, want)):
            assert float((a.float() - b.float()).norm() / b.float().norm()) <= 2.0 ** -7


@pytest.mark.parametrize("name", FORMS)
def test_a_decoder_that_routes_keeps_its_roundings(name, monkeypatch):
    """A router turns another rounding into another expert: its decoder's heads are rounded where the separate kernels round them."""
    part = _layer(FORMS[name])
    formed, out, k, v = _step(part, monkeypatch, separate=False, routed=True)
    _, want, k2, v2 = _step(part, monkeypatch, separate=True, routed=True)
    assert formed == (1 if name in SAME_BITS else 0)
    assert torch.equal(k, k2) and torch.equal(v, v2) and torch.equal(out, want)


@pytest.mark.parametrize("name", SEPARATE)
def test_what_the_attention_does_not_form(name, monkeypatch):
    assert _step(_layer(SEPARATE[name]), monkeypatch, separate=False, writes_cache=SEPARATE[name].get("own_kv", True))[0] == 0


@pytest.mark.parametrize("array", ["bias", "angles", "norms"])
def test_arrays_off_a_boundary_go_to_the_separate_kernels(array, monkeypatch):
    part = _layer({"bias": dict(qkv_bias=True), "angles": {}, "norms": dict(qk_norm_eps=1e-5)}[array])
    _, want, k, v = _step(part, monkeypatch, separate=True)
    if array == "bias":
        part.b_qkv = _off(part.b_qkv, 1)
    if array == "norms":
        part.k_norm = _off(part.k_norm, 3)
    formed, out, k2, v2 = _step(part, monkeypatch, separate=False, shift=2 if array == "angles" else 0)
    assert formed == 0 and torch.equal(out, want) and torch.equal(k, k2) and torch.equal(v, v2)


def test_a_position_encoding_of_ones_own_keeps_its_interface(monkeypatch):
    """A registered encoding whose methods know nothing of an attention that forms heads is called as it was, and one that changes a
    method of the rotary one is not passed by."""
    from rust_inference_b200.parts.registry import lookup, register, unregister
    base = lookup("position", "rope")
    called = []

    @register("position", "toy_rope")
    class Toy(base):
        def apply_and_store_from_accumulators(self, acc, bias, q_out, ctx, cache_layer, *, n_heads, n_kv_heads, head_dim, write_kv):
            called.append("sums")
            super().apply_and_store_from_accumulators(acc, bias, q_out, ctx, cache_layer, n_heads=n_heads, n_kv_heads=n_kv_heads,
                                                      head_dim=head_dim, write_kv=write_kv)

        def apply_and_store(self, *args, **kw):
            called.append("rows")
            super().apply_and_store(*args, **kw)

    try:
        for form, way in (({}, "sums"), (dict(rot_dims=64), "rows")):
            _, want, k, v = _step(_layer(form), monkeypatch, separate=True)
            called.clear()
            formed, out, k2, v2 = _step(_layer(form, kind="toy_rope"), monkeypatch, separate=False)
            assert formed == 0 and called == [way]
            assert torch.equal(out, want) and torch.equal(k, k2) and torch.equal(v, v2)
    finally:
        unregister("position", "toy_rope")


@pytest.mark.parametrize("graphs", [True, False])
def test_an_engine_decodes_over_a_page_edge(graphs, monkeypatch):
    """Steps of a dense decoder from before a page's edge to behind it: every layer's attention forms its heads, and the logits are
    those of the separate kernels."""
    from rust_inference_b200 import Engine, config_from_dict
    from rust_inference_b200.kernels import attention
    config = config_from_dict({
        "architectures": ["Qwen2ForCausalLM"], "hidden_size": 1024, "num_hidden_layers": 3, "num_attention_heads": 8, "num_key_value_heads": 2,
        "head_dim": 128, "intermediate_size": 512, "vocab_size": 264, "rope_theta": 1e6, "rms_norm_eps": 1e-6, "attention_bias": True,
        "tie_word_embeddings": False, "max_position_embeddings": 512})
    tokens = [[(7 * i + 3 * b) % 264 for i in range(70)] for b in range(2)]
    rows, counts = [], []
    real, rule = attention.FormedHeads.run, attention.formed_heads
    for separate in (False, True):
        runs = []
        monkeypatch.setattr(attention.FormedHeads, "run", lambda self, *a, **k: (runs.append(1), real(self, *a, **k))[1])
        monkeypatch.setattr(attention, "formed_heads", (lambda *a, **k: None) if separate else rule)
        eng = Engine.from_random(config, std=0.03, max_tokens=1024, n_slots=3, use_graphs=graphs)
        slots = [eng.alloc_slot(), eng.alloc_slot()]
        eng.step(slots, [t[:62 - b] for b, t in enumerate(tokens)], "none")
        got = [eng.step(slots, [[t[62 - b + i]] for b, t in enumerate(tokens)], "last").clone() for i in range(6)]
        torch.cuda.synchronize()
        eng.check_device_status()
        rows.append(torch.cat(got))
        counts.append(len(runs))
    # a captured step passes here when it is warmed up and captured, the others every time
    assert counts[1] == 0 and counts[0] % 3 == 0 and counts[0] >= (3 if graphs else 18)
    # the same sums and roundings but for the order in which pieces of K are added
    assert float((rows[0] - rows[1]).norm() / rows[1].norm()) <= 1e-2
