"""The decode attention that forms the new position's heads from the sums of their projection, against the kernels that do so step
by step."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _case(lengths, nh, nkv, hd, rot, from_keys, seed):
    """Sums, cache filled with older positions, and the step's arrays; lengths count the new position."""
    from rust_inference_b200.parts.rope import rope_tables
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, pages = len(lengths), 6
    width = (nh + (1 if from_keys else 2) * nkv) * hd
    acc = torch.randn(n, width, device=DEV, generator=g)
    bias = torch.randn(width, device=DEV, generator=g)
    k, v = (torch.randn(n * pages + 1, nkv, 64, hd, device=DEV, generator=g).bfloat16() for _ in range(2))
    table = torch.randperm(n * pages, generator=torch.Generator().manual_seed(seed)).int().view(n, pages).to(DEV)
    cos, sin = (torch.from_numpy(t).to(DEV) for t in rope_tables(rot, 10000.0, pages * 64))
    step = dict(page_table=table, seq_slot=_i32(list(range(n))), seq_len=_i32(list(lengths)), cu_seqlens=_i32(list(range(n + 1))))
    return acc, bias, k, v, cos, sin, step


@pytest.mark.parametrize("nh, nkv, hd, rot, style, normed, from_keys, window, splits", [
    (14, 2, 64, 64, 0, False, False, 0, 8), (28, 4, 128, 128, 0, False, False, 0, 3), (16, 1, 128, 128, 1, False, False, 0, 1),
    (2, 2, 64, 32, 1, False, False, 0, 2), (16, 4, 128, 64, 0, False, False, -128, 4), (8, 2, 128, 64, 1, True, True, 100, 2),
    (6, 2, 64, 8, 0, True, False, 0, 1), (32, 2, 128, 128, 0, True, True, 64, 8)])
def test_heads_formed_in_the_attention(nh, nkv, hd, rot, style, normed, from_keys, window, splits):
    from rust_inference_b200.kernels import attention_tc, ops, tcgen05
    lengths = [1, 2, 63, 64, 65, 128, 129, 200, 384]
    n = len(lengths)
    acc, bias, k, v, cos, sin, step = _case(lengths, nh, nkv, hd, rot, from_keys, seed=nh + hd + rot)
    qw, kw = (torch.rand(hd, device=DEV) + 0.5 for _ in range(2)) if normed else (None, None)
    # step by step, in float32: bias, norm, rotation, one rounding to bfloat16
    z = (acc + bias).view(n, -1, hd)
    heads, values = z[:, :nh + nkv], z[:, nh:nh + nkv] if from_keys else z[:, nh + nkv:]
    if normed:
        inv = 1.0 / torch.sqrt((heads * heads).mean(-1, keepdim=True) + 1e-5)
        heads = heads * inv * torch.cat([qw.expand(nh, hd), kw.expand(nkv, hd)])
    pos = torch.tensor(lengths, device=DEV) - 1
    c, s = cos[pos][:, None], sin[pos][:, None]
    turned = heads.clone()
    a, b = (heads[..., 0:rot:2], heads[..., 1:rot:2]) if style else (heads[..., :rot // 2], heads[..., rot // 2:rot])
    at = (slice(0, rot, 2), slice(1, rot, 2)) if style else (slice(0, rot // 2), slice(rot // 2, rot))
    turned[..., at[0]], turned[..., at[1]] = a * c - b * s, a * s + b * c
    q = turned[:, :nh].reshape(n, -1).bfloat16().contiguous()
    k2, v2 = k.clone(), v.clone()
    for i, length in enumerate(lengths):
        page = step["page_table"][i, (length - 1) // 64].long()
        k2[page, :, (length - 1) % 64] = turned[i, nh:].bfloat16()
        v2[page, :, (length - 1) % 64] = values[i].bfloat16()
    sizes = dict(n_seqs=n, n_heads=nh, n_kv_heads=nkv, head_dim=hd, page_size=64, scale=hd ** -0.5, window=window)
    want = torch.empty(n, nh * hd, device=DEV, dtype=torch.bfloat16)
    kernel = attention_tc.decode if splits == 1 else attention_tc.decode_cluster
    kernel(q, nh * hd, k2, v2, step["page_table"], step["seq_slot"], step["seq_len"], step["cu_seqlens"], want, n_splits=splits, **sizes)
    got = torch.full_like(want, 9.0)
    attention_tc.decode_form(acc, bias, cos, sin, qw, kw, 1e-5, k, v, step["page_table"], step["seq_slot"], step["seq_len"],
                             step["cu_seqlens"], got, n_splits=splits, style=style, rot_dims=rot, values_from_keys=from_keys,
                             out_scale=0.5, **sizes)
    torch.cuda.synchronize()
    tcgen05.check_status()
    assert float(acc.abs().max()) == 0.0                                  # left zeroed
    # one bfloat16 step where float32 sums in another order round to the other side
    for mine, theirs in ((k, k2), (v, v2)):
        assert ((mine.float() - theirs.float()).abs() <= theirs.float().abs() * 2.0 ** -7 + 1e-30).all()
    # a result is a mean of values of about 1 with weights in bfloat16: heads that differ by one rounding (2^-8) move it by less than that
    assert float((2.0 * got.float() - want.float()).abs().max()) <= 2.0 ** -6 * float(want.float().abs().max())


def test_formed_heads_keep_infinities_where_they_are():
    """Channels that are not turned pass as they are: an infinite value channel makes no NaN."""
    from rust_inference_b200.kernels import attention_tc
    acc, bias, k, v, cos, sin, step = _case([5, 70], 4, 2, 64, 32, False, seed=3)
    acc[0, 6 * 64 + 3] = float("inf")                                     # the first kv head's value, channel 3
    out = torch.empty(2, 4 * 64, device=DEV, dtype=torch.bfloat16)
    attention_tc.decode_form(acc, bias, cos, sin, None, None, 0.0, k, v, step["page_table"], step["seq_slot"], step["seq_len"],
                             step["cu_seqlens"], out, n_splits=2, style=0, rot_dims=32, n_seqs=2, n_heads=4, n_kv_heads=2, head_dim=64,
                             page_size=64, scale=0.125, window=0)
    odd = ~torch.isfinite(out.float())
    assert torch.isposinf(out[0, [3, 64 + 3]].float()).all() and int(odd.sum()) == 2
