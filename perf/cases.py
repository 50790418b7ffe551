"""The work that this library is timed on: decode steps and prompts of dense decoders in both run precisions, and of two
of the other architectures (routed experts beside a gated linear recurrence; attention over a window and over a latent).

Every case builds a whole model from seeded random tensors, keeps it with its cache as a serving program does, and runs
one step of the engine per pass: token ids in from the host, float32 logits out on the device.

    listed()            the cases
    draw(rng)           one more of the same ranges
    prepare(case, seed) model, cache (filled, for a decode step) and token ids
    run(state)          one pass
    work(case)          the bytes and operations a pass cannot do without
    tolerance(case)     how far another correct implementation at the same precision may be off
    exact(case, seed)   the same logits in 64 bits by plain torch
"""
from __future__ import annotations

import math
import random
import zlib

import torch

DEVICE = "cuda:0"
ROOM = 4096                     # decode steps a cache has room for behind the prompts before they are filled in again
GROUP = 8                       # prompts that go into one step when a decode case's cache is filled


def _dense(hidden, layers, heads, kv, head_dim, ff, vocab, theta, eps, bias, tied):
    return {"architectures": ["Qwen2ForCausalLM" if bias else "LlamaForCausalLM"], "hidden_size": hidden,
            "num_hidden_layers": layers, "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": head_dim,
            "intermediate_size": ff, "vocab_size": vocab, "rope_theta": theta, "rms_norm_eps": eps, "attention_bias": bias,
            "tie_word_embeddings": tied, "max_position_embeddings": 32768}


def _lulisun(width, layers, heads, kv, hd, chunk, rot, rheads, experts, top, ff, groups, keep, shared, vocab):
    layer = {"type": "parallel", "mixer": {
        "left": {"heads": heads, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": 1.0 / math.sqrt(hd), "mask": {"size": chunk},
                 "rot": {"base": 10000.0, "dims": rot}},
        "right": {"heads": rheads, "dim": hd, "vdim": hd}, "left_scale": 0.7, "right_scale": 0.7},
        "mlp": {"kind": "moe", "expert": {"ff": ff},
                "router": {"experts": experts, "top": top, "groups": {"count": groups, "keep": keep}}, "shared": {"ff": shared}}}
    return {"architecture": "Lulisun", "vocab": vocab, "width": width, "norm": {"eps": 1e-5}, "layers": [layer] * layers}


def _vadodra(width, heads, kv, hd, window, rot, lheads, ldim, lrot, lvdim, rank, ff, vocab):
    mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
    near = {"type": "attention", "mlp": mlp, "mixer": {
        "heads": heads, "kv_heads": kv, "dim": hd, "vdim": hd, "scale": 1.0 / math.sqrt(hd), "mask": {"size": window},
        "rot": {"base": 500000.0, "dims": rot, "scaling": {"factor": 4.0}}}}
    lat = {"heads": lheads, "dim": ldim, "rot_dim": lrot, "vdim": lvdim, "kv_rank": rank, "scale": 1.0 / math.sqrt(ldim + lrot),
           "rot": {"base": 10000.0, "dims": lrot}}
    return {"architecture": "Vadodra", "vocab": vocab, "width": width, "norm": {"eps": 1e-5},
            "embedding": {"scale": math.sqrt(width)},
            "layers": [near, {"type": "latent_attention", "mixer": lat, "mlp": mlp}, near,
                       {"type": "latent_attention", "mixer": {**lat, "kv_from": 1}, "mlp": mlp}]}


# the layer sizes that bench.py runs
MODELS = {
    "qwen2-0.5b": _dense(896, 24, 14, 2, 64, 4864, 151936, 1e6, 1e-6, True, True),
    "qwen2-1.5b": _dense(1536, 28, 12, 2, 128, 8960, 151936, 1e6, 1e-6, True, True),
    "qwen2.5-3b": _dense(2048, 36, 16, 2, 128, 11008, 151936, 1e6, 1e-6, True, True),
    "qwen2.5-7b": _dense(3584, 28, 28, 4, 128, 18944, 152064, 1e6, 1e-6, True, False),
    "llama3-8b": _dense(4096, 32, 32, 8, 128, 14336, 128256, 5e5, 1e-5, False, False),
    "lulisun-1k": _lulisun(1024, 4, 8, 2, 128, 512, 64, 4, 16, 2, 512, 4, 2, 1024, 32000),
    "lulisun-2k": _lulisun(2048, 4, 16, 4, 128, 1024, 64, 8, 32, 4, 512, 8, 4, 2048, 32000),
    "vadodra-1k": _vadodra(1024, 8, 2, 128, 512, 64, 8, 128, 64, 128, 256, 4096, 32000),
    "vadodra-2k": _vadodra(2048, 16, 4, 128, 1024, 64, 16, 128, 64, 128, 512, 8192, 32000),
}


def _case(name, model, dtype, kind, batch, shortest, longest, logits="last"):
    case = {"model": model, "dtype": dtype, "pass": kind, "sequences": batch, "shortest": shortest, "longest": longest,
            "logits": logits}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user waiting for the next token of a small model: the smallest step, bound by its chain of launches
        _case("decode 0.5b x1", "qwen2-0.5b", "bfloat16", "decode", 1, 437, 437),
        # a server's ordinary step: the benchmark model, eight sequences of unequal length
        _case("decode 7b x8", "qwen2.5-7b", "bfloat16", "decode", 8, 128, 2048),
        # a full batch of a mid-sized model
        _case("decode 3b x64", "qwen2.5-3b", "bfloat16", "decode", 64, 128, 1500),
        # one prompt of the benchmark's length, its next token wanted
        _case("prompt 7b 2048", "qwen2.5-7b", "bfloat16", "prompt", 1, 2048, 2048),
        # a handful of short and odd prompts that arrived together
        _case("prompts 1.5b x7", "qwen2-1.5b", "bfloat16", "prompt", 7, 9, 611),
        # a long document, the largest single call
        _case("prompt 8b 7999", "llama3-8b", "bfloat16", "prompt", 1, 7999, 7999),
        # the 32-bit run of a small model: a step of a few sequences
        _case("decode 1.5b x4 f32", "qwen2-1.5b", "float32", "decode", 4, 100, 700),
        # the 32-bit run of a prompt, logits at every position (scoring a text)
        _case("prompt 0.5b 333 f32", "qwen2-0.5b", "float32", "prompt", 1, 333, 333, "all"),
        # routed experts, a gated recurrence and attention over chunks: a prompt and a step
        _case("prompt lulisun 2048", "lulisun-2k", "bfloat16", "prompt", 1, 2048, 2048),
        _case("decode lulisun x8", "lulisun-2k", "bfloat16", "decode", 8, 700, 1280),
        # attention over a window and over a shared latent: a prompt and a step
        _case("prompt vadodra 2048", "vadodra-2k", "bfloat16", "prompt", 1, 2048, 2048),
        _case("decode vadodra x8", "vadodra-2k", "bfloat16", "decode", 8, 700, 1280),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "prompt"])
    family = rng.choice(["dense", "dense", "dense", "float32", "lulisun", "vadodra"])
    if family == "dense":
        model, most_sequences, most_tokens = rng.choice([("qwen2-0.5b", 64, 7999), ("qwen2-1.5b", 64, 7999), ("qwen2.5-3b", 64, 7999),
                                                         ("qwen2.5-7b", 24, 7999), ("llama3-8b", 24, 7999)])
    elif family == "float32":
        model, most_sequences, most_tokens = rng.choice([("qwen2-0.5b", 16, 512), ("qwen2-1.5b", 8, 256)])
    else:
        model, most_sequences, most_tokens = rng.choice([(family + "-1k", 32, 4096), (family + "-2k", 32, 4096)])
    dtype = "float32" if family == "float32" else "bfloat16"
    if kind == "decode":
        n = _log(rng, 1, most_sequences)
        longest = _log(rng, 32, 1500)
        return _case(None, model, dtype, kind, n, max(1, longest // rng.randint(1, 12)), longest)
    total = _log(rng, 12, most_tokens)
    n = min(total, rng.choice([1, 1, 2, 3, 5, 8]))
    longest = max(1, total // n)
    wanted = "all" if dtype == "float32" and n == 1 and rng.random() < 0.5 else "last"
    return _case(None, model, dtype, kind, n, max(1, longest // rng.randint(1, 12)), longest, wanted)


def _lengths(case):
    """The sequences' lengths: fixed by the case, the first one the longest."""
    rng = random.Random("%(sequences)d %(shortest)d %(longest)d" % case)
    return [case["longest"]] + [rng.randint(case["shortest"], case["longest"]) for _ in range(case["sequences"] - 1)]


def _tokens(case, seed):
    """Per sequence its prompt and, for a decode case, the ids that its steps are fed."""
    cfg = MODELS[case["model"]]
    vocab = cfg.get("vocab_size", cfg.get("vocab"))
    rng = random.Random(seed * 7919 + 1)
    prompts = [[rng.randrange(vocab) for _ in range(n)] for n in _lengths(case)]
    steps = [[[rng.randrange(vocab)] for _ in prompts] for _ in range(64)] if case["pass"] == "decode" else []
    return prompts, steps


# ---- tensors ------------------------------------------------------------------------------------------------------
def _shapes(cfg):
    """name -> (shape, kind): "matrix" (N(0, 1 / inputs)), "out" (a branch's last matrix: smaller by the root of the number of
    branches, as trained decoders start from), "embed", "norm" (around 1), "offset" (around 0), "bias", "unit" (in 0..0.9)."""
    out = {}
    if "architectures" in cfg:
        d, hd, ff = cfg["hidden_size"], cfg["head_dim"], cfg["intermediate_size"]
        q, kv = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd
        out["model.embed_tokens.weight"] = ((cfg["vocab_size"], d), "embed")
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            out[p + "input_layernorm.weight"] = ((d,), "norm")
            for n, rows in (("q", q), ("k", kv), ("v", kv)):
                out[p + f"self_attn.{n}_proj.weight"] = ((rows, d), "matrix")
                if cfg["attention_bias"]:
                    out[p + f"self_attn.{n}_proj.bias"] = ((rows,), "bias")
            out[p + "self_attn.o_proj.weight"] = ((d, q), "out")
            out[p + "post_attention_layernorm.weight"] = ((d,), "norm")
            out[p + "mlp.gate_proj.weight"] = ((ff, d), "matrix")
            out[p + "mlp.up_proj.weight"] = ((ff, d), "matrix")
            out[p + "mlp.down_proj.weight"] = ((d, ff), "out")
        out["model.norm.weight"] = ((d,), "norm")
        if not cfg["tie_word_embeddings"]:
            out["lm_head.weight"] = ((cfg["vocab_size"], d), "matrix")
        return out
    d = cfg["width"]
    out["embed"] = ((cfg["vocab"], d), "embed")
    if cfg["architecture"] == "Lulisun":
        out["final.norm"] = ((d,), "offset")
        out["head"] = ((cfg["vocab"], d), "matrix")
        for i, layer in enumerate(cfg["layers"]):
            p, left, right, mlp = f"l{i}.", layer["mixer"]["left"], layer["mixer"]["right"], layer["mlp"]
            out[p + "norm1"] = out[p + "norm2"] = ((d,), "offset")
            out[p + "mix.left.q"] = ((left["heads"] * left["dim"], d), "matrix")
            out[p + "mix.left.k"] = ((left["kv_heads"] * left["dim"], d), "matrix")
            out[p + "mix.left.v"] = ((left["kv_heads"] * left["vdim"], d), "matrix")
            out[p + "mix.left.o"] = ((d, left["heads"] * left["vdim"]), "out")
            rows = right["heads"] * right["dim"]
            out[p + "mix.right.q"] = out[p + "mix.right.f"] = ((rows, d), "matrix")
            out[p + "mix.right.f.b"] = ((rows,), "bias")
            out[p + "mix.right.lower"] = ((rows,), "unit")
            out[p + "mix.right.v"] = ((right["heads"] * right["vdim"], d), "matrix")
            out[p + "mix.right.norm"] = ((right["vdim"],), "norm")
            out[p + "mix.right.o"] = ((d, right["heads"] * right["vdim"]), "out")
            widths = [(f"mlp.e{e}.", mlp["expert"]["ff"]) for e in range(mlp["router"]["experts"])] + [("mlp.shared.", mlp["shared"]["ff"])]
            for e, ff in widths:
                out[p + e + "gate"] = out[p + e + "up"] = ((ff, d), "matrix")
                out[p + e + "down"] = ((d, ff), "out")
            out[p + "mlp.router"] = ((mlp["router"]["experts"], d), "matrix")
            out[p + "mlp.correction"] = ((mlp["router"]["experts"],), "bias")
            out[p + "mlp.shared.sg"] = ((1, d), "matrix")
        return out
    out["final.norm"] = ((d,), "norm")
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        out[p + "norm1"] = ((d,), "norm")
        if layer["type"] == "attention":
            out[p + "mix.q"] = ((m["heads"] * m["dim"], d), "matrix")
            out[p + "mix.k"] = ((m["kv_heads"] * m["dim"], d), "matrix")
            out[p + "mix.q.norm"] = out[p + "mix.k.norm"] = ((m["dim"],), "norm")
        else:
            out[p + "mix.q"] = ((m["heads"] * (m["dim"] + m["rot_dim"]), d), "matrix")
            if m.get("kv_from") is None:
                out[p + "mix.dkv"] = ((m["kv_rank"] + m["rot_dim"], d), "matrix")
                out[p + "mix.dkv.norm"] = ((m["kv_rank"],), "norm")
            out[p + "mix.uk"] = ((m["heads"] * m["dim"], m["kv_rank"]), "matrix")
            out[p + "mix.uv"] = ((m["heads"] * m["vdim"], m["kv_rank"]), "matrix")
            out[p + "mix.g"] = ((m["heads"], d), "matrix")
        out[p + "mix.o"] = ((d, m["heads"] * m["vdim"]), "out")
        out[p + "mlp.gate"] = out[p + "mlp.up"] = ((ff, d), "matrix")
        out[p + "mlp.down"] = ((d, ff), "out")
    return out


def _weights(case, seed):
    """(name, tensor) pairs on the GPU: matrices in the run precision, vectors in float32."""
    cfg = MODELS[case["model"]]
    dtype = getattr(torch, case["dtype"])
    branches = 2 * (cfg["num_hidden_layers"] if "architectures" in cfg else len(cfg["layers"]))
    scale = cfg.get("embedding", {}).get("scale", 1.0)
    gen = torch.Generator(device=DEVICE)
    for name, (shape, kind) in _shapes(cfg).items():
        gen.manual_seed(zlib.crc32(f"{seed} {name}".encode()))
        t = torch.empty(shape, dtype=dtype if len(shape) == 2 else torch.float32, device=DEVICE)
        if kind == "unit":
            t.uniform_(0.0, 0.9, generator=gen)
        else:
            std = {"matrix": 1.0 / math.sqrt(shape[-1]), "out": 1.0 / math.sqrt(shape[-1] * branches), "embed": 1.0 / scale}.get(kind, 0.1)
            t.normal_(1.0 if kind == "norm" else 0.0, std, generator=gen)
        yield name, t


# ---- a pass -------------------------------------------------------------------------------------------------------
class _State:
    def __init__(self, case, model, prompts, steps):
        self.case, self.model, self.prompts, self.steps = case, model, prompts, steps
        self.slots, self.done = [], 0

    def fill(self):
        """Prompts into the cache: new slots, a few prompts per step."""
        engine = self.model.engine
        for slot in self.slots:
            engine.free_slot(slot)
        self.slots, self.done = [engine.alloc_slot() for _ in self.prompts], 0
        for i in range(0, len(self.slots), GROUP):
            engine.step(self.slots[i:i + GROUP], self.prompts[i:i + GROUP], "none")


def prepare(case, seed):
    from rust_inference_b200 import Engine, Model, config_from_dict
    from rust_inference_b200.config.registry import get_architecture
    from rust_inference_b200.engine.model import DecoderModel
    prompts, steps = _tokens(case, seed)
    room = ROOM if case["pass"] == "decode" else 64
    tokens = sum(-(-(len(p) + room) // 64) * 64 for p in prompts)
    positions = 8192
    while positions < case["longest"] + room:
        positions *= 2
    config = config_from_dict(MODELS[case["model"]])
    decoder = DecoderModel(get_architecture(config.architecture).build_spec(config), dtype=getattr(torch, case["dtype"]), device=DEVICE)
    decoder.load(_weights(case, seed))
    state = _State(case, Model(Engine(decoder, max_tokens=max(tokens, positions), max_seq_len=positions, n_slots=len(prompts) + 1)),
                   prompts, steps)
    if case["pass"] == "decode":
        state.fill()
    return state


def run(state):
    engine = state.model.engine
    if state.case["pass"] == "decode":
        if state.done == ROOM:
            state.fill()
        logits = engine.step(state.slots, state.steps[state.done % len(state.steps)], "last")
        state.done += 1
        return logits
    if len(state.prompts) == 1:
        return state.model.logits(state.prompts[0], state.case["logits"])
    slots = [engine.alloc_slot() for _ in state.prompts]
    logits = engine.step(slots, state.prompts, state.case["logits"])
    for slot in slots:
        engine.free_slot(slot)
    return logits


def _spans(cfg):
    """Per layer: (keys a query sees at most, values cached per position, multiply-adds per visible key)."""
    if "architectures" in cfg:
        hd = cfg["head_dim"]
        return [(None, 2 * cfg["num_key_value_heads"] * hd, 2 * cfg["num_attention_heads"] * hd)] * cfg["num_hidden_layers"]
    out = []
    for layer in cfg["layers"]:
        m = layer["mixer"]
        if layer["type"] == "parallel":
            m = m["left"]
            out.append((m["mask"]["size"], 2 * m["kv_heads"] * m["dim"], 2 * m["heads"] * m["dim"]))
        elif layer["type"] == "attention":
            out.append((m["mask"]["size"], 2 * m["kv_heads"] * m["dim"], 2 * m["heads"] * m["dim"]))
        else:       # a key of each head has dim + rot_dim channels, its value vdim; a position is cached once for all heads
            out.append((None, m["kv_rank"] + m["rot_dim"], m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])))
    return out


def work(case):
    cfg = MODELS[case["model"]]
    item = 4 if case["dtype"] == "float32" else 2
    lengths = _lengths(case)
    decode = case["pass"] == "decode"
    tokens = len(lengths) if decode else sum(lengths)
    rows = tokens if case["logits"] == "all" else len(lengths)
    tied = cfg.get("tie_word_embeddings", cfg.get("architecture") == "Vadodra")
    bytes_, flops = 0.0, 0.0
    router = None if "architectures" in cfg or cfg["layers"][0]["mlp"].get("router") is None else cfg["layers"][0]["mlp"]["router"]
    for name, (shape, kind) in _shapes(cfg).items():
        n = math.prod(shape)
        if kind == "embed":
            bytes_ += tokens * shape[1] * item
            if tied:
                bytes_, flops = bytes_ + n * item, flops + 2.0 * n * rows
        elif ".mlp.e" in name:      # a routed expert: a token passes `top` of them, a step reads those that are chosen
            share = router["top"] / router["experts"]
            bytes_ += n * item * min(1.0, 1.0 - (1.0 - share) ** tokens)
            flops += 2.0 * n * tokens * share
        else:
            bytes_ += n * (item if len(shape) == 2 else 4)
            if len(shape) == 2:
                flops += 2.0 * n * (rows if name in ("lm_head.weight", "head") else tokens)
    vocab = cfg.get("vocab_size", cfg.get("vocab"))
    bytes_ += 4.0 * rows * vocab
    for span, cached, macs in _spans(cfg):
        for n in lengths:
            if decode:
                seen = min(n + 1, span or n + 1)
                bytes_, flops = bytes_ + seen * cached * item, flops + 2.0 * seen * macs
            else:
                near = min(n, span or n)
                pairs = near * (near + 1) / 2 + (n - near) * near
                bytes_, flops = bytes_ + n * cached * item, flops + 2.0 * pairs * macs
    if cfg.get("architecture") == "Lulisun":
        for layer in cfg["layers"]:
            r = layer["mixer"]["right"]
            state = r["heads"] * r["dim"] * r["vdim"]
            bytes_, flops = bytes_ + len(lengths) * state * 4 * (2 if decode else 1), flops + 5.0 * state * tokens
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # measured against exact(): 0.9e-6 to 1.2e-6 in float32, 2.0e-3 to 4.5e-3 in bfloat16 (the same step twice: up to 2.8e-3,
    # since pieces of a split sum are added in no fixed order)
    return {"rel": 5e-6} if case["dtype"] == "float32" else {"rel": 1e-2}


# ---- the same logits in 64 bits -------------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _turn(x, base, dims, adjacent=False, factor=1.0):
    """x [T, heads, d]: the first `dims` channels of every head turned by their position's angles, in halves or adjacent pairs."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    a = torch.arange(len(x), dtype=torch.float64, device=x.device)[:, None] * (float(base) ** (-2.0 * i / dims) / factor)[None]
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    at = (slice(0, dims, 2), slice(1, dims, 2)) if adjacent else (slice(0, dims // 2), slice(dims // 2, dims))
    out = x.clone()
    u, v = x[..., at[0]], x[..., at[1]]
    out[..., at[0]], out[..., at[1]] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, window=None, chunk=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv]: causal, over a window of positions or inside chunks of them, head by head."""
    t, h = len(q), q.shape[1]
    pos = torch.arange(t, device=q.device)
    hidden = pos[None] > pos[:, None]
    if window is not None:
        hidden |= pos[None] <= pos[:, None] - window
    if chunk is not None:
        hidden |= pos[None] // chunk != pos[:, None] // chunk
    out = torch.empty(t, h, v.shape[2], dtype=q.dtype, device=q.device)
    for i in range(h):
        g = i // (h // k.shape[1])
        s = (q[:, i] @ k[:, g].T).mul_(scale).masked_fill_(hidden, -math.inf)
        out[:, i] = torch.softmax(s, -1) @ v[:, g]
    return out.reshape(t, -1)


def _exact_dense(cfg, w, ids):
    eps, hd, heads, kv = cfg["rms_norm_eps"], cfg["head_dim"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
    x = w["model.embed_tokens.weight"][ids]
    t = len(ids)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, w[p + "input_layernorm.weight"], eps)
        q, k, v = (h @ w[p + f"self_attn.{n}_proj.weight"].T + w.get(p + f"self_attn.{n}_proj.bias", 0.0) for n in "qkv")
        q, k = (_turn(z.view(t, -1, hd), cfg["rope_theta"], hd) for z in (q, k))
        x = x + _attend(q, k, v.view(t, kv, hd), hd ** -0.5) @ w[p + "self_attn.o_proj.weight"].T
        h = _rms(x, w[p + "post_attention_layernorm.weight"], eps)
        gate = torch.nn.functional.silu(h @ w[p + "mlp.gate_proj.weight"].T)
        x = x + (gate * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
    x = _rms(x, w["model.norm.weight"], eps)
    return x, w["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]


def _exact_lulisun(cfg, w, ids):
    eps, t = cfg["norm"]["eps"], len(ids)
    silu = torch.nn.functional.silu
    x = w["embed"][ids]
    for i, layer in enumerate(cfg["layers"]):
        p, left, right, mlp = f"l{i}.", layer["mixer"]["left"], layer["mixer"]["right"], layer["mlp"]
        h = _rms(x, 1.0 + w[p + "norm1"], eps)
        q, k, v = (h @ w[p + "mix.left." + n].T for n in "qkv")
        q, k = (_turn(z.view(t, -1, left["dim"]), left["rot"]["base"], left["rot"]["dims"]) for z in (q, k))
        a = _attend(q, k, v.view(t, -1, left["vdim"]), left["scale"], chunk=left["mask"]["size"]) @ w[p + "mix.left.o"].T
        low = w[p + "mix.right.lower"]
        f = low + (1.0 - low) * torch.sigmoid(h @ w[p + "mix.right.f"].T + w[p + "mix.right.f.b"])
        f, q = f.view(t, right["heads"], -1, 1), silu(h @ w[p + "mix.right.q"].T).view(t, right["heads"], 1, -1)
        v = (h @ w[p + "mix.right.v"].T).view(t, right["heads"], 1, -1)
        state = torch.zeros(right["heads"], right["dim"], right["vdim"], dtype=x.dtype, device=x.device)
        o = torch.empty_like(v)
        for n in range(t):
            state = torch.addcmul((1.0 - f[n]) * v[n], f[n], state)
            torch.matmul(q[n], state, out=o[n])
        r = _rms(o[:, :, 0], w[p + "mix.right.norm"], eps).reshape(t, -1) @ w[p + "mix.right.o"].T
        y = layer["mixer"]["left_scale"] * a + layer["mixer"]["right_scale"] * r
        h, router = _rms(x, 1.0 + w[p + "norm2"], eps), mlp["router"]
        score = torch.sigmoid(h @ w[p + "mlp.router"].T)
        choice = (score + w[p + "mlp.correction"]).view(t, router["groups"]["count"], -1)
        best = choice.topk(2, -1).values.sum(-1).topk(router["groups"]["keep"], -1).indices
        kept = torch.zeros(choice.shape[:2], dtype=torch.bool, device=x.device).scatter_(1, best, True)
        chosen = choice.masked_fill(~kept[..., None], -math.inf).view(t, -1).topk(router["top"], -1).indices
        share = torch.zeros_like(score).scatter_(1, chosen, score.gather(1, chosen))
        share = share / share.sum(-1, keepdim=True)
        for e in range(router["experts"]):
            at = share[:, e].nonzero()[:, 0]
            z, pre = h[at], p + f"mlp.e{e}."
            y.index_add_(0, at, share[at, e, None] * ((silu(z @ w[pre + "gate"].T) * (z @ w[pre + "up"].T)) @ w[pre + "down"].T))
        pre = p + "mlp.shared."
        x = x + y + torch.sigmoid(h @ w[pre + "sg"].T) * ((silu(h @ w[pre + "gate"].T) * (h @ w[pre + "up"].T)) @ w[pre + "down"].T)
    return _rms(x, 1.0 + w["final.norm"], eps), w["head"]


def _exact_vadodra(cfg, w, ids):
    eps, t = cfg["norm"]["eps"], len(ids)

    def centred(x, weight):
        d = x - x.mean(-1, keepdim=True)
        return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * weight

    x, rows = w["embed"][ids] * cfg["embedding"]["scale"], None
    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        h, rot = centred(x, w[p + "norm1"]), m["rot"]
        if layer["type"] == "attention":
            q, v = ((h @ w[p + "mix." + n].T).view(t, -1, m["dim"]) for n in "qk")
            q, k = (_turn(_rms(z, w[p + f"mix.{n}.norm"], eps), rot["base"], rot["dims"], True, rot["scaling"]["factor"])
                    for n, z in (("q", q), ("k", v)))
            mixed = _attend(q, k, v, m["scale"], window=m["mask"]["size"])
        else:
            rank, d = m["kv_rank"], m["dim"]
            if m.get("kv_from") is None:
                down = h @ w[p + "mix.dkv"].T
                rows = _rms(down[:, :rank], w[p + "mix.dkv.norm"], eps), _turn(down[:, None, rank:], rot["base"], rot["dims"])
            q = (h @ w[p + "mix.q"].T).view(t, m["heads"], -1)
            q = torch.cat([q[..., :d], _turn(q[..., d:], rot["base"], rot["dims"])], -1)
            k = torch.cat([(rows[0] @ w[p + "mix.uk"].T).view(t, m["heads"], d), rows[1].expand(-1, m["heads"], -1)], -1)
            v = (rows[0] @ w[p + "mix.uv"].T).view(t, m["heads"], -1)
            mixed = _attend(q, k, v, m["scale"]).view(t, m["heads"], -1) * torch.sigmoid(h @ w[p + "mix.g"].T)[..., None]
            mixed = mixed.reshape(t, -1)
        limit = layer["mlp"]["limit"]
        g = torch.clamp(h @ w[p + "mlp.gate"].T, max=limit)
        u = torch.clamp(h @ w[p + "mlp.up"].T, -limit, limit)
        x = x + mixed @ w[p + "mix.o"].T + (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[p + "mlp.down"].T
    return centred(x, w["final.norm"]), w["embed"]


def exact(case, seed):
    cfg = MODELS[case["model"]]
    prompts, steps = _tokens(case, seed)
    if case["pass"] == "decode":
        prompts = [p + t for p, t in zip(prompts, steps[0])]
    layers = {"Lulisun": _exact_lulisun, "Vadodra": _exact_vadodra}.get(cfg.get("architecture"), _exact_dense)
    with torch.no_grad():
        w = {name: t.double() for name, t in _weights(case, seed)}
        out = []
        for p in prompts:
            x, head = layers(cfg, w, torch.tensor(p, device=DEVICE))
            out.append((x if case["logits"] == "all" else x[-1:]) @ head.T)
        return torch.cat(out)
