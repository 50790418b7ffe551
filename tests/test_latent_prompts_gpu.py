"""Prompts through latent attention with keys and values formed head by head (heads of 128 + 64 key and 128 value channels)."""
import math

import pytest
import torch

import plain_vadodra
from conftest import TOL, random_tokens, rel_err

pytestmark = pytest.mark.gpu


def _config(heads, rank, style_layers, vocab=515):
    mlp = {"kind": "dense", "ff": 320, "limit": 7.0}
    lat = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": rank, "scale": 1.0 / math.sqrt(192),
           "rot": {"base": 10000.0, "dims": 64}}
    layers = []
    for i, source in enumerate(style_layers):
        mixer = lat if source is None else {**lat, "kv_from": source}
        layers.append({"type": "latent_attention", "mixer": mixer, "mlp": mlp})
    return {"architecture": "Vadodra", "vocab": vocab, "width": 256, "norm": {"eps": 1e-5}, "embedding": {"scale": 16.0}, "layers": layers}


@pytest.mark.parametrize("heads, rank", [(8, 64), (16, 512), (8, 256)])          # gated rows of whole 16-byte pieces
@pytest.mark.parametrize("lengths", [[2], [64], [65], [1, 129, 63], [300, 128]])
def test_prompts(heads, rank, lengths, monkeypatch):
    """Every position's logits of prompts around the edges of pages (64) and query tiles (128), alone and side by side, against
    the plain form; a layer with a latent of its own, another one, and one that reads the first one's rows.  Then the next
    tokens, which read the cache that the prompts left."""
    from rust_inference_b200 import config_from_dict
    from rust_inference_b200.config.registry import get_architecture
    from rust_inference_b200.engine.engine import Engine
    from rust_inference_b200.engine.model import DecoderModel
    from rust_inference_b200.kernels import attention_tc
    cfg = _config(heads, rank, [None, None, 0])
    config = config_from_dict(cfg)
    weights = plain_vadodra.random_weights(cfg, seed=heads)
    model = DecoderModel(get_architecture(config.architecture).build_spec(config), dtype=torch.bfloat16, device="cuda")
    model.load(weights.items())
    eng = Engine(model, max_tokens=2048, max_seq_len=1024, n_slots=4)
    taken = []
    expanded = attention_tc.expanded
    monkeypatch.setattr(attention_tc, "expanded", lambda *a, **k: taken.append(1) or expanded(*a, **k))
    prompts = [random_tokens(n, cfg["vocab"], seed=n) for n in lengths]
    slots = [eng.alloc_slot() for _ in prompts]
    got = eng.step(slots, prompts, "all")
    assert len(taken) == 3
    more = [random_tokens(1, cfg["vocab"], seed=90 + n) for n in lengths]
    after = eng.step(slots, more, "last")
    eng.check_device_status()
    assert len(taken) == 3                                     # single tokens read the cached rows
    at = 0
    for i, (p, m) in enumerate(zip(prompts, more)):
        want = plain_vadodra.forward(cfg, weights, p + m)
        assert rel_err(got[at:at + len(p)], want[:len(p)]) <= TOL["bfloat16"]
        assert rel_err(after[i:i + 1], want[-1:]) <= TOL["bfloat16"]
        at += len(p)


@pytest.mark.parametrize("window, sink, gated", [(0, False, False), (50, False, True), (130, True, True), (0, True, False)])
@pytest.mark.parametrize("lengths", [[1, 200], [64, 65, 128], [333]])
def test_kernel(window, sink, gated, lengths):
    """The attention alone against 64 bits: windows, a sink and gates."""
    from rust_inference_b200.kernels import attention_tc, tcgen05
    heads, total = 3, sum(lengths)
    g = torch.Generator(device="cuda").manual_seed(total)
    draw = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    q, kv, shared, gates = draw(total, heads * 192 + 16), draw(total, heads * 256), draw(total, 64), draw(total, 8)
    sinks = torch.randn(heads, device="cuda", generator=g) if sink else None
    cu = torch.tensor([sum(lengths[:i]) for i in range(len(lengths) + 1)], dtype=torch.int32, device="cuda")
    zeros = torch.zeros(len(lengths), dtype=torch.int32, device="cuda")
    out = torch.empty(total, heads * 128, dtype=torch.bfloat16, device="cuda")
    attention_tc.expanded(q, kv, shared, zeros, zeros, cu, out, n_seqs=len(lengths), max_new=max(lengths), n_heads=heads,
                          scale=192 ** -0.5, window=window, sink=sinks, gate=gates[:, 2:2 + heads] if gated else None)
    torch.cuda.synchronize()
    tcgen05.check_status()
    at = 0
    for n in lengths:
        rows = slice(at, at + n)
        pos = torch.arange(n, device="cuda")
        hidden = pos[None] > pos[:, None]
        if window:
            hidden |= pos[None] <= pos[:, None] - window
        for h in range(heads):
            k = torch.cat([kv[rows, h * 256:h * 256 + 128], shared[rows]], 1).double()
            s = (q[rows, h * 192:(h + 1) * 192].double() @ k.T * 192 ** -0.5).masked_fill(hidden, -math.inf)
            if sink:
                s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
            want = torch.softmax(s, 1)[:, :n] @ kv[rows, h * 256 + 128:(h + 1) * 256].double()
            if gated:
                want = want * torch.sigmoid(gates[rows, 2 + h].double())[:, None]
            # probabilities and results are rounded to bfloat16 (2^-9 each)
            got = out[rows, h * 128:(h + 1) * 128].double()
            assert (got - want).abs().max().item() <= 2 ** -7 * want.abs().max().item()
        at += n


@pytest.mark.parametrize("first", [1, 63, 65, 130, 200])         # the last page holds 63, 1, 63, 62 and 56 rows of the next prompt
@pytest.mark.parametrize("gated, terms", [(False, 1), (True, 1), (False, 2)])
def test_neighbours_with_infinities(first, gated, terms):
    """A prompt's result does not depend on what stands in the prompt packed behind it, infinities and NaN included: to the
    bit what it is alone."""
    from rust_inference_b200.kernels import attention_tc, tcgen05
    heads, second = 3, 100
    g = torch.Generator(device="cuda").manual_seed(first)
    draw = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    total = first + second
    q, kv, shared, gates = draw(total, heads * 192), draw(total, heads * 256), draw(total, 64), draw(total, 8)
    low = draw(total, heads * 128) * 2.0 ** -8 if terms == 2 else None
    for t in (q, kv, shared) + ((low,) if terms == 2 else ()):
        t[first::3], t[first + 1::3], t[first + 2::3] = float("nan"), float("inf"), float("-inf")

    def run(n, lengths):
        cu = torch.tensor([sum(lengths[:i]) for i in range(len(lengths) + 1)], dtype=torch.int32, device="cuda")
        zeros = torch.zeros(len(lengths), dtype=torch.int32, device="cuda")
        out = torch.full((n, heads * 128), 7.0, dtype=torch.bfloat16, device="cuda")
        attention_tc.expanded(q[:n], kv[:n], shared[:n], zeros, zeros, cu, out, n_seqs=len(lengths), max_new=max(lengths), n_heads=heads,
                              scale=192 ** -0.5, gate=gates[:n, 2:2 + heads] if gated else None, low=low[:n] if terms == 2 else None)
        torch.cuda.synchronize()
        tcgen05.check_status()
        return out

    alone, beside = run(first, [first]), run(total, [first, second])
    assert bool(alone.isfinite().all())
    assert torch.equal(beside[:first], alone)


@pytest.mark.parametrize("lengths", [[2], [16, 5], [70, 128]])
def test_values_in_two_terms(lengths):
    """Short prompts hold a value as the sum of two bfloat16 numbers: the float32 values come back to 2^-16, and the attention over
    them is as close to 64 bits over the float32 values as its rounded weights and result (2^-8 each at most) allow; where a
    token sees one key (weight 1), only the result is rounded."""
    from rust_inference_b200.kernels import attention_tc, ops, tcgen05
    heads, total = 3, sum(lengths)
    g = torch.Generator(device="cuda").manual_seed(total)
    kv32 = torch.randn(total, heads * 256, device="cuda", generator=g)
    q, shared = (torch.randn(total, n, device="cuda", generator=g).bfloat16() for n in (heads * 192, 64))
    kv, low = torch.empty(total, heads * 256, dtype=torch.bfloat16, device="cuda"), torch.empty(total, heads * 128, dtype=torch.bfloat16, device="cuda")
    ops.latent_terms(kv32, kv, low, n_heads=heads, head_dim=128, v_head_dim=128)
    assert torch.equal(kv, kv32.bfloat16())
    values = kv32.view(total, heads, 256)[:, :, 128:].double()
    terms = kv.view(total, heads, 256)[:, :, 128:].double() + low.view(total, heads, 128).double()
    assert ((terms - values).abs() <= 2.0 ** -16 * values.abs()).all()
    cu = torch.tensor([sum(lengths[:i]) for i in range(len(lengths) + 1)], dtype=torch.int32, device="cuda")
    zeros = torch.zeros(len(lengths), dtype=torch.int32, device="cuda")
    out = torch.empty(total, heads * 128, dtype=torch.bfloat16, device="cuda")
    attention_tc.expanded(q, kv, shared, zeros, zeros, cu, out, n_seqs=len(lengths), max_new=max(lengths), n_heads=heads,
                          scale=192 ** -0.5, low=low)
    torch.cuda.synchronize()
    tcgen05.check_status()
    at = 0
    for n in lengths:
        rows = slice(at, at + n)
        hidden = torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1)
        for h in range(heads):
            k = torch.cat([kv[rows, h * 256:h * 256 + 128], shared[rows]], 1).double()
            s = (q[rows, h * 192:(h + 1) * 192].double() @ k.T * 192 ** -0.5).masked_fill(hidden, -math.inf)
            want = torch.softmax(s, 1) @ values[rows, h]
            got = out[rows, h * 128:(h + 1) * 128].double()
            assert ((got[0] - want[0]).abs() <= 2.0 ** -8 * (1 + 2.0 ** -7) * want[0].abs()).all()
            assert (got - want).abs().max().item() <= 2 ** -7 * want.abs().max().item()
        at += n


def test_short_prompts_take_two_terms(monkeypatch):
    """The shortest prompt of a step decides."""
    from rust_inference_b200 import config_from_dict
    from rust_inference_b200.config.registry import get_architecture
    from rust_inference_b200.engine.engine import Engine
    from rust_inference_b200.engine.model import DecoderModel
    from rust_inference_b200.kernels import attention_tc
    cfg = _config(8, 64, [None])
    config = config_from_dict(cfg)
    model = DecoderModel(get_architecture(config.architecture).build_spec(config), dtype=torch.bfloat16, device="cuda")
    model.load(plain_vadodra.random_weights(cfg, seed=1).items())
    eng = Engine(model, max_tokens=2048, max_seq_len=1024, n_slots=4)
    taken = []
    expanded = attention_tc.expanded
    monkeypatch.setattr(attention_tc, "expanded", lambda *a, **k: taken.append(k["low"] is not None) or expanded(*a, **k))
    for lengths in ([255], [256], [300, 256], [300, 2]):
        slots = [eng.alloc_slot() for _ in lengths]
        eng.step(slots, [random_tokens(n, cfg["vocab"], seed=n) for n in lengths], "last")
        for slot in slots:
            eng.free_slot(slot)
    eng.check_device_status()
    assert taken == [True, False, False, True]
