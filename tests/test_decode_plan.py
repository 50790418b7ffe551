"""Which decode-attention kernel a step takes and into how many runs it cuts a sequence
(`kernels.attention.decode_plan`): decided on the host from the batch size, the cache geometry and what
the device says it can hold, so it is tested here with a device that is made up."""
import pytest


@pytest.fixture
def plan(monkeypatch):
    from rust_inference_b200.kernels import attention, attention_tc
    monkeypatch.setattr(attention, "_sm_count", lambda: 148)
    monkeypatch.setattr(attention, "_DECODE", "auto")
    monkeypatch.delenv("RI_B200_DECODE_SPLITS", raising=False)
    held = {}

    def capacity(head_dim, n_splits):
        return held["fn"](head_dim, n_splits)
    monkeypatch.setattr(attention_tc, "decode_cluster_capacity", capacity)

    def run(n_seqs, n_kv_heads, max_seq_len, head_dim=None, fits=lambda hd, s: 10 ** 6):
        held["fn"] = fits
        return attention.decode_plan(n_seqs, n_kv_heads, max_seq_len, 64, head_dim)
    return run


def test_small_batches_take_clusters_and_large_ones_whole_sequences(plan, monkeypatch):
    assert plan(1, 4, 8192) == ("cluster", 8)            # 4 pairs: eight runs each, the most a cluster holds
    assert plan(8, 4, 8192) == ("cluster", 8)            # 32 pairs x 8 = 256 CTAs <= two per SM
    assert plan(16, 4, 8192) == ("cluster", 4)
    assert plan(32, 4, 8192) == ("cluster", 2)
    assert plan(37, 4, 8192) == ("cluster", 2)           # 148 pairs x 2 = 296
    assert plan(38, 4, 8192) == ("tma", 1)
    assert plan(64, 4, 8192) == ("tma", 1)
    assert plan(1, 4, 64) == ("tma", 1)                  # one page per sequence: nothing to cut
    assert plan(1, 4, 200) == ("cluster", 4)             # never more runs than pages


def test_runs_are_made_fewer_until_the_step_is_resident_together(plan):
    # what a B200 answers for head size 128: clusters of 2..8 CTAs it holds at once
    b200 = {2: 148, 3: 93, 4: 71, 5: 56, 6: 45, 7: 37, 8: 33}
    fits = lambda hd, s: b200[s]
    assert plan(8, 4, 8192, 128, fits) == ("cluster", 8)         # 32 clusters of eight fit (33)
    assert plan(9, 4, 8192, 128, fits) == ("cluster", 7)         # 36 clusters: seven CTAs each (37)
    assert plan(16, 4, 8192, 128, fits) == ("cluster", 4)
    # a device that holds fewer: the runs shrink; with no room for clusters at all the runs are merged
    # through scratch by a second kernel
    assert plan(8, 4, 8192, 128, lambda hd, s: 40 if s <= 4 else 8) == ("cluster", 4)
    assert plan(8, 4, 8192, 128, lambda hd, s: 8) == ("tma", 9)
    # without a head size nobody is asked
    assert plan(8, 4, 8192, None, lambda hd, s: 0) == ("cluster", 8)


def test_the_kernel_can_be_forced(plan, monkeypatch):
    from rust_inference_b200.kernels import attention
    monkeypatch.setattr(attention, "_DECODE", "cp_async")
    assert plan(8, 4, 8192) == ("cp_async", 9)
    assert plan(64, 4, 8192) == ("cp_async", 1)
    monkeypatch.setattr(attention, "_DECODE", "tma")
    assert plan(8, 4, 8192) == ("tma", 9)


def test_float32_attention_leaves_to_the_generic_kernel_what_the_tiles_do_not_take(monkeypatch):
    """More sequences than a launch grid's third axis holds, caches that are no whole aligned 16-byte pieces, other pages and heads."""
    from types import SimpleNamespace

    import torch
    from rust_inference_b200.kernels import attention, ops
    monkeypatch.setattr(attention, "_sm_count", lambda: 148)
    taken = []
    monkeypatch.setattr(ops, "attention_f32", lambda *a, **k: taken.append("tiles"))
    monkeypatch.setattr(ops, "attention_generic", lambda *a, **k: taken.append("generic"))

    def route(n_seqs=2, kv=2, hd=64, page=64, offset=0):
        floats = torch.zeros(3 * kv * page * hd + 64)
        floats = floats[-(floats.data_ptr() // 4) % 4:]            # a 16-byte boundary
        k = floats[offset:offset + 3 * kv * page * hd].view(3, kv, page, hd)
        q = torch.zeros(4, 2 * kv * hd)
        none = torch.zeros(1, dtype=torch.int32)
        ctx = SimpleNamespace(n_seqs=n_seqs, max_new=1, max_len=100, all_single=True, page_size=page, page_table=torch.zeros(2, 3),
                              token_pos=none, token_seq=none, seq_slot=none, seq_start=none, cu_seqlens=none)
        taken.clear()
        attention.attention(q, SimpleNamespace(k=k, v=k), torch.zeros_like(q), ctx, n_heads=2 * kv, n_kv_heads=kv, head_dim=hd, scale=0.1)
        return taken[0]

    assert route() == route(hd=128) == route(n_seqs=65535) == route(offset=4) == "tiles"
    assert route(n_seqs=65536) == route(offset=1) == route(hd=80) == route(page=32) == "generic"


def test_float32_prompts_of_few_keys_stay_with_the_generic_kernel(monkeypatch):
    """Where a tile's fixed time is longer than a block per token and head takes for its few keys."""
    from types import SimpleNamespace

    import torch
    from rust_inference_b200.kernels import attention, ops
    monkeypatch.setattr(attention, "_sm_count", lambda: 148)
    taken = []
    monkeypatch.setattr(ops, "attention_f32", lambda *a, **k: taken.append("tiles"))
    monkeypatch.setattr(ops, "attention_generic", lambda *a, **k: taken.append("generic"))
    monkeypatch.setattr(ops, "attention_f32_supports", lambda *a, **k: True)

    def route(new, cached=0, seqs=1, heads=12, kv=2, single=False):
        none = torch.zeros(1, dtype=torch.int32)
        q = torch.zeros(new * seqs, 1)
        ctx = SimpleNamespace(n_seqs=seqs, max_new=new, max_len=new + cached, all_single=single, page_size=64,
                              page_table=torch.zeros(2, 1), token_pos=none, token_seq=none, seq_slot=none, seq_start=none, cu_seqlens=none)
        taken.clear()
        attention.attention(q, SimpleNamespace(k=q, v=q), q, ctx, n_heads=heads, n_kv_heads=kv, head_dim=128, scale=0.1)
        return taken[0]

    assert [route(n) for n in (2, 3, 32, 33, 64)] == ["tiles", "generic", "generic", "tiles", "tiles"]     # 12 rows: the kernel for few
    assert [route(3, cached=c) for c in (29, 30)] == ["generic", "tiles"]
    assert [route(24, seqs=n) for n in (4, 5)] == ["generic", "tiles"]             # 1,152 and 1,440 blocks on 8 x 148
    assert route(1, heads=40, kv=2, single=True) == "tiles"                        # a captured step: by the cache's geometry
    assert route(16, heads=8, kv=8) == "tiles" and route(17, heads=8, kv=8) == "generic"


def test_short_float32_sums_stay_with_the_ffma_kernel(monkeypatch):
    import torch
    from rust_inference_b200.kernels import linear, ops
    monkeypatch.setattr(linear, "_sm_count", lambda: 148)
    taken = []
    monkeypatch.setattr(ops, "gemm_f32", lambda *a, **k: taken.append("parts"))
    monkeypatch.setattr(ops, "gemm_simt", lambda *a, **k: taken.append("ffma"))

    def route(m, n, k):
        taken.clear()
        linear._plain(torch.zeros(m, k), linear.Weight(torch.zeros(n, k)), torch.zeros(m, n), ops.EPI_STORE)
        return taken[0]

    assert [route(16, 512, k) for k in (4, 128, 2048)] == ["parts"] * 3            # few rows: a kernel of their own
    assert [route(17, 512, k) for k in (124, 128, 256)] == ["ffma", "parts", "parts"]
    assert [route(33, 512, k) for k in (128, 252, 256)] == ["ffma", "ffma", "parts"]
    assert [route(333, n, 128) for n in (512, 24 * 64, 25 * 64)] == ["ffma", "ffma", "parts"]      # 6 x 24 = 144 tiles, 150
    assert route(333, 512, 130) == route(333, 512, 2050) == "ffma"                  # rows of no whole 16-byte pieces
