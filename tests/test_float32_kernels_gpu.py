"""The kernels of the 32-bit path alone: products by a few rows and by many (operands in three bfloat16 parts on the tensor
cores) and attention in tiles of query rows, at the edges of their tiles."""
import random

import pytest
import torch

import plain_impl

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ops():
    from rust_inference_b200.kernels import ops
    return ops


def _check_status():
    from rust_inference_b200.kernels import tcgen05
    torch.cuda.synchronize()
    tcgen05.check_f32_status()


@pytest.mark.parametrize("few_max", [-1, 0])          # the default choice; the tensor cores for few rows too
@pytest.mark.parametrize("m", [1, 2, 3, 8, 9, 16, 17, 32, 33, 64, 65, 128, 130, 300])
@pytest.mark.parametrize("n, k", [(7, 4), (100, 36), (391, 192), (130, 1032), (1152, 896), (264, 4864)])
def test_product(m, n, k, few_max):
    """Every epilogue against 64 bits.  The bound: a float32 sum of k products, each rounded (2^-24 of the running sum),
    errs by about 2^-24 sqrt(k) of a typical result, and the largest of m n results lies a few times above typical;
    2e-6 of the largest is what the FFMA kernel's test asks for."""
    ops = _ops()
    torch.manual_seed(m * 1000 + n)
    x = torch.randn(m, k, device=DEV) * 0.5
    w = torch.randn(n, k, device=DEV) * 0.1
    w2 = torch.randn(n, k, device=DEV) * 0.1
    bias = torch.randn(n, device=DEV)
    ref, ref2 = x.double() @ w.double().t(), x.double() @ w2.double().t()
    scale = ref.abs().max().item()
    assert ops.gemm_f32_supports(x, w, w2)

    def run(mode, start=None, **kw):
        out = torch.full((m, n), 9.0, device=DEV) if start is None else start.clone()
        ops.gemm_f32(x, w, out, mode, few_max=few_max, **kw)
        again = torch.full((m, n), 7.0, device=DEV) if start is None else start.clone()
        ops.gemm_f32(x, w, again, mode, few_max=few_max, **kw)
        assert torch.equal(out, again)                                     # sums in a fixed order
        return out.double()

    assert (run(ops.EPI_STORE, bias=bias) - (ref + bias)).abs().max().item() <= 2e-6 * (scale + bias.abs().max().item())
    assert (run(ops.EPI_STORE_F32) - ref).abs().max().item() <= 2e-6 * scale
    before = torch.randn(m, n, device=DEV)
    assert (run(ops.EPI_RESIDUAL, start=before) - (before + ref)).abs().max().item() <= 2e-6 * (scale + 4)
    want = plain_impl.silu(ref) * ref2
    assert (run(ops.EPI_SILU_MUL, w2=w2) - want).abs().max().item() <= 4e-6 * (want.abs().max().item() + 1e-3)
    cols = torch.tensor([float(n // 2)], device=DEV)
    want = torch.cat([plain_impl.silu(ref[:, :n // 2]), ref[:, n // 2:]], 1)
    assert (run(ops.EPI_SILU_F32, silu_cols=cols) - want).abs().max().item() <= 2e-6 * (scale + 1e-3)
    form = torch.tensor(ops.RELU_SQUARED_FORM, device=DEV)
    want = ref.clamp_min(0) ** 2
    assert (run(ops.EPI_ACT, act_form=form) - want).abs().max().item() <= 4e-6 * (want.abs().max().item() + 1e-3)
    _check_status()


@pytest.mark.parametrize("m", [3, 40, 200])
def test_product_with_infinities(m):
    """Infinite and NaN operands come out as the plain float32 sum gives them, and leave other rows alone."""
    ops = _ops()
    torch.manual_seed(5)
    x, w = torch.randn(m, 640, device=DEV), torch.randn(200, 640, device=DEV)
    clean = torch.empty(m, 200, device=DEV)
    ops.gemm_f32(x, w, clean, ops.EPI_STORE_F32)
    x[1, 100], x[2, 600] = float("inf"), float("nan")
    w[3, 630] = float("-inf")
    x[0, 0] = 3e38                        # its product with most weights overflows
    w[4, :] = 0.0
    got, want = torch.empty(m, 200, device=DEV), torch.empty(m, 200, device=DEV)
    ops.gemm_f32(x, w, got, ops.EPI_STORE_F32)
    ops.gemm_simt(x, w, want, ops.EPI_STORE_F32)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[got.isinf()])
    rows = [r for r in range(3, m)]
    cols = [c for c in range(200) if c not in (3, 4)]
    if rows:
        assert (got[rows][:, cols] - clean[rows][:, cols]).abs().max().item() <= 2e-6 * clean.abs().max().item()
    _check_status()


@pytest.mark.parametrize("m, n, k", [(20, 200, 640), (40, 130, 100), (200, 200, 640), (130, 391, 4864)])
@pytest.mark.parametrize("mode", ["store", "gated"])
def test_product_keeps_finite_sums_beside_infinite_ones(mode, m, n, k):
    """Sums that do not meet an infinity, a NaN or an overflow keep their bits; those that do come out as the plain float32 sum's
    infinities and NaN.  Rows and features at the matrices' ends, whose tiles are filled up with zeros, are among them."""
    ops = _ops()
    torch.manual_seed(m)
    x, w, w2 = torch.randn(m, k, device=DEV), torch.randn(n, k, device=DEV), torch.randn(n, k, device=DEV)

    def run(kernel, **kw):
        out = torch.full((m, n), 9.0, device=DEV)
        if mode == "gated":
            kernel(x, w, out, ops.EPI_SILU_MUL, w2=w2, **kw)
        else:
            kernel(x, w, out, ops.EPI_STORE_F32, **kw)
        return out

    clean = run(ops.gemm_f32, few_max=0)
    rows, cols = [1, 2, m - 1], [3, n - 1]
    x[1, k // 3], x[2, k - 1], x[m - 1, 0] = float("inf"), float("nan"), 3e38
    w[3, k - 2], w[n - 1, 5] = float("-inf"), float("nan")
    got, want = run(ops.gemm_f32, few_max=0), run(ops.gemm_simt)
    _check_status()
    same = torch.ones(m, n, dtype=torch.bool, device=DEV)
    same[rows] = False
    same[:, cols] = False
    assert torch.equal(got[same], clean[same])
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[got.isinf()])


def test_product_with_small_and_large_numbers():
    """Three parts hold a float32 number over its whole range: scaling the operands by powers of two scales the result."""
    ops = _ops()
    torch.manual_seed(6)
    x, w = torch.randn(130, 256, device=DEV), torch.randn(140, 256, device=DEV)
    base, out = torch.empty(130, 140, device=DEV), torch.empty(130, 140, device=DEV)
    ops.gemm_f32(x, w, base, ops.EPI_STORE_F32)
    for up, down in ((2.0 ** 100, 2.0 ** -60), (2.0 ** -80, 2.0 ** 70)):
        ops.gemm_f32(x * up, w * down, out, ops.EPI_STORE_F32)
        assert torch.equal(out, base * (up * down))
    _check_status()


def _operands(kind, m, n, k, gen):
    """Rows of x and of w: dense ones of either or of one sign, numbers whose lower 16 bits are all set (nothing of them is in a first
    bfloat16 part), rows with few entries, squared rectified ones, and numbers down to the denormal ones."""
    draw = lambda *s: torch.randn(*s, device=DEV, generator=gen)
    if kind == "positive":
        return torch.rand(m, k, device=DEV, generator=gen), torch.rand(n, k, device=DEV, generator=gen)
    if kind == "full mantissas":
        return tuple((torch.randint(0x3f80ff00, 0x3f810000, s, device=DEV, generator=gen, dtype=torch.int32).view(torch.float32))
                     for s in ((m, k), (n, k)))
    w = draw(n, k)
    if kind.startswith("entries"):
        keep = torch.rand(m, k, device=DEV, generator=gen).argsort(1)[:, :int(kind.split()[1])]
        return torch.zeros(m, k, device=DEV).scatter_(1, keep, draw(m, k)), w
    if kind == "squared":
        return draw(m, k).clamp_min(0) ** 2, w
    if kind.startswith("2^"):
        return (draw(m, k).double() * 2.0 ** int(kind[2:])).float(), w * 2.0 ** 20
    return draw(m, k), w


@pytest.mark.parametrize("m, n, k", [(20, 264, 128), (130, 264, 896), (40, 130, 4864)])
@pytest.mark.parametrize("kind", ["dense", "positive", "full mantissas", "entries 1", "entries 2", "entries 4", "entries 16", "squared",
                                  "2^-100", "2^-112", "2^-120", "2^-130", "2^-140"])
def test_product_in_parts_is_as_close_as_the_plain_sum(kind, m, n, k):
    """Cutting operands into bfloat16 parts costs no accuracy, whatever is in the rows: against 64 bits the root mean square of
    the errors stays below that of the FFMA kernel's (for rows of a few entries, whose terms that one rounds together with the
    sum and a sum in blocks each for itself, below 1.25 of it), and no result leans to one side by more than one truncated addition
    of the tensor core, 2^-23.  A single product is rounded once (2^-24), but for what is left out of it (2^-30) and
    truncated of its small parts (2^-23 of 2^-7)."""
    ops = _ops()
    x, w = _operands(kind, m, n, k, torch.Generator(device=DEV).manual_seed(m))
    ref = x.double() @ w.double().t()
    got, plain = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    ops.gemm_f32(x, w, got, ops.EPI_STORE_F32, few_max=0)
    ops.gemm_simt(x, w, plain, ops.EPI_STORE_F32)
    _check_status()
    error, error_plain = got.double() - ref, plain.double() - ref
    few = kind.startswith("entries") and int(kind.split()[1]) < 16
    assert error.norm() <= (1.25 if few else 1.0) * error_plain.norm()
    assert (error * ref.sign()).mean().abs() <= 2.0 ** -23 * ref.abs().mean()
    if kind == "entries 1":
        assert (error.abs() <= 2.0 ** -24 * (1 + 2.0 ** -4) * ref.abs()).all()


@pytest.mark.parametrize("splits", [1, 2, 5, 8])
@pytest.mark.parametrize("span", [0, 50, -96])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("heads, kv, starts, news", [
    (14, 2, [0], [333]), (6, 2, [100, 0, 63, 700], [1, 1, 1, 1]), (8, 8, [5, 0], [70, 3]), (12, 2, [100, 0, 200], [40, 130, 1]),
    (40, 2, [10, 300], [1, 1]), (16, 1, [127, 128, 0], [1, 1, 1])])
def test_attention(hd, heads, kv, starts, news, span, splits):
    """Against the generic kernel, which visits the same keys one by one; places beyond a sequence's end hold NaN."""
    ops = _ops()
    rng = random.Random(hd + heads + splits)
    torch.manual_seed(heads)
    need = [-(-(s + n) // 64) for s, n in zip(starts, news)]
    order = list(range(sum(need) + 2))
    rng.shuffle(order)
    slots = list(range(len(starts)))
    rng.shuffle(slots)
    table = torch.zeros(len(starts), max(need), dtype=torch.int32)
    kc, vc = torch.randn(len(order), kv, 64, hd), torch.randn(len(order), kv, 64, hd)
    for b, pages in enumerate(need):
        for j in range(pages):
            table[slots[b], j] = order.pop()
        end = starts[b] + news[b]
        if end % 64:
            last = int(table[slots[b], end // 64])
            kc[last, :, end % 64:] = vc[last, :, end % 64:] = float("nan")
    total = sum(news)
    d = lambda t, kind=torch.int32: torch.as_tensor(t, dtype=kind).to(DEV)
    kc, vc, table = kc.to(DEV), vc.to(DEV), table.to(DEV)
    q = torch.randn(total, heads * hd + 8, device=DEV)
    pos = d([s + i for s, n in zip(starts, news) for i in range(n)])
    seq = d([b for b, n in enumerate(news) for _ in range(n)])
    cu = d([sum(news[:i]) for i in range(len(news) + 1)])
    slot, start = d(slots), d(starts)
    want, got = torch.empty(total, heads * hd, device=DEV), torch.full((total, heads * hd), 7.0, device=DEV)
    common = dict(n_heads=heads, n_kv_heads=kv, head_dim=hd, page_size=64, scale=hd ** -0.5, out_scale=0.7)
    ops.attention_generic(q, q.shape[1], kc, vc, table, pos, seq, slot, want, n_tokens=total, window=max(span, 0),
                          chunk=max(-span, 0), **common)
    ops.attention_f32(q, q.shape[1], kc, vc, table, slot, start, cu, got, n_seqs=len(news), max_new=max(news), span=span,
                      n_splits=splits, **common)
    # two float32 sums over at most 701 keys in different orders
    assert (got - want).abs().max().item() <= 5e-6 * want.abs().max().item()


@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("heads, kv, start, new", [(6, 2, 150, 1), (4, 4, 20, 3), (14, 2, 0, 200)])
def test_attention_with_infinite_values(hd, heads, kv, start, new, splits):
    """A value that is infinite or NaN reaches every row that sees its key, also where the key's weight is so small that it is 0
    (0 times an infinity is NaN), and no other row: as in the generic kernel, which visits the seen keys only."""
    ops = _ops()
    torch.manual_seed(hd + heads)
    end, page = start + new, 64
    pages = -(-end // page)
    kc, vc = torch.randn(pages, kv, page, hd), torch.randn(pages, kv, page, hd)
    kc[0, :, 9] = -40.0                        # its scores lie hundreds below the others'
    vc[0, 0, 9, 5], vc[0, -1, 9, 7] = float("inf"), float("nan")
    if new > 100:
        vc[1, 0, 50, 2] = float("-inf")         # seen by the later rows, with an ordinary weight
    q = torch.randn(new, heads * hd).abs() + 1.0
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    table, slot, first = i32([list(range(pages))]), i32([0]), i32([start])
    kc, vc, q = kc.to(DEV), vc.to(DEV), q.to(DEV)
    want, got = torch.empty(new, heads * hd, device=DEV), torch.full((new, heads * hd), 7.0, device=DEV)
    common = dict(n_heads=heads, n_kv_heads=kv, head_dim=hd, page_size=page, scale=hd ** -0.5)
    ops.attention_generic(q, q.shape[1], kc, vc, table, i32(list(range(start, end))), i32([0] * new), slot, want, n_tokens=new, **common)
    ops.attention_f32(q, q.shape[1], kc, vc, table, slot, first, i32([0, new]), got, n_seqs=1, max_new=new, n_splits=splits, **common)
    assert bool(want.isnan().any()) and not bool(want.isnan().all())
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    fine = want.isfinite()
    assert (got[fine] - want[fine]).abs().max().item() <= 5e-6 * want[fine].abs().max().item()
