"""Float32 products of many rows whose rows are cut into their parts in memory, at the edges of their tiles, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ops():
    from rust_inference_b200.kernels import ops
    return ops


@pytest.mark.parametrize("m, n, k", [(1, 7, 4), (65, 130, 260), (128, 128, 64), (129, 200, 68), (333, 300, 576), (500, 64, 2052)])
@pytest.mark.parametrize("tile, splits", [(0, 0), (16, 1), (48, 2), (112, 1), (128, 8)])
def test_wide_products_at_the_edges_of_their_tiles(m, n, k, tile, splits):
    ops = _ops()
    from rust_inference_b200.kernels import tcgen05
    blocks = -(-k // 64)
    splits = min(splits, 1 << (blocks.bit_length() - 1))
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x = torch.randn(m, k, device=DEV, generator=g)
    w, w2 = (torch.randn(n, k, device=DEV, generator=g) / k ** 0.5 for _ in range(2))
    bias = torch.randn(n, device=DEV, generator=g)
    ref, ref2 = x.double() @ w.double().t(), x.double() @ w2.double().t()
    # a sum of 64 steps is off by 2^-22 of its operands' size at most, and every block adds one rounding of the sum so far
    tol = (4 + blocks) * 2.0 ** -24
    cut = dict(tile=tile, splits=splits)
    out = torch.full((m, n), 9.0, device=DEV)
    ops.gemm_f32_wide(x, w, out, ops.EPI_STORE, bias=bias, **cut)
    assert float((out.double() - ref - bias).norm() / ref.norm()) <= tol + 2.0 ** -23
    act = torch.full((m, n), 9.0, device=DEV)
    ops.gemm_f32_wide(x, w, act, ops.EPI_SILU_MUL, w2=w2, **cut)
    want = ref * torch.sigmoid(ref) * ref2
    assert float((act.double() - want).norm() / want.norm()) <= 2 * tol + 2.0 ** -21
    res = torch.ones(m, n, device=DEV)
    ops.gemm_f32_wide(x, w, res, ops.EPI_RESIDUAL, **cut)
    assert float((res.double() - 1 - ref).norm() / ref.norm()) <= tol + 2.0 ** -22
    torch.cuda.synchronize()
    tcgen05.check_f32_status()


@pytest.mark.parametrize("splits", [1, 4])
def test_wide_products_with_infinities_keep_their_neighbours(splits):
    ops = _ops()
    m, n, k = 150, 200, 320
    x, w = torch.randn(m, k, device=DEV), torch.randn(n, k, device=DEV)
    clean = torch.empty(m, n, device=DEV)
    ops.gemm_f32_wide(x, w, clean, ops.EPI_STORE_F32, tile=80, splits=splits)
    x[3, 7], x[149, 319], w[130, 100], w[199, 0] = float("inf"), float("nan"), -float("inf"), 3e38
    got, want = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    ops.gemm_f32_wide(x, w, got, ops.EPI_STORE_F32, tile=80, splits=splits)
    ops.gemm_simt(x, w, want, ops.EPI_STORE_F32)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isposinf(got), torch.isposinf(want))
    rows, cols = [i for i in range(m) if i not in (3, 149)], [j for j in range(n) if j not in (130, 199)]
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols])


@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("size", [0.0, 2.0 ** -70, 2.0 ** -50, 2.0 ** -48])
def test_wide_products_add_to_subnormal_numbers(size, splits):
    """Sums of nothing, of 2^-140, and on both sides of 2^-100, added to subnormal numbers and to what nearly cancels them."""
    ops = _ops()
    x, w = torch.zeros(70, 192, device=DEV), torch.zeros(130, 192, device=DEV)
    x[:, 0], w[:, 0] = size, size * 1.25
    v = torch.tensor(size).float() * (size * 1.25)
    out = torch.full((70, 130), 2.0 ** -139, device=DEV)
    out[:, 1::3], out[:, 2::3] = 3 * 2.0 ** -149, -v.item() * (1.0 + 2.0 ** -23)
    want = out.cpu().clone() + v
    ops.gemm_f32_wide(x, w, out, ops.EPI_RESIDUAL, splits=splits)
    assert torch.equal(out.cpu(), want)


@pytest.mark.parametrize("m, rows", [(300, 128), (257, 256), (100, 1), (64, 64), (300, 299)])
def test_wide_products_in_stretches_of_rows(m, rows):
    """Fewer rows of scratch than x has: cut and multiplied a stretch at a time, with the sums of the whole."""
    ops = _ops()
    n, k = 200, 260
    x, w = torch.randn(m, k, device=DEV), torch.randn(n, k, device=DEV) / 16
    whole, out = torch.ones(m, n, device=DEV), torch.ones(m + 1, n, device=DEV)
    ops.gemm_f32_wide(x, w, whole, ops.EPI_RESIDUAL, splits=1)
    parts = torch.empty(3, rows, 264, device=DEV, dtype=torch.bfloat16)
    ops.gemm_f32_wide(x, w, out[:m], ops.EPI_RESIDUAL, splits=1, parts=parts)
    assert torch.equal(out[:m], whole) and bool((out[m] == 1).all())


def test_the_scratch_of_wide_products_is_bounded():
    ops = _ops()
    for m, k in ((8000, 18944), (100000, 896), (500, 262144), (70, 64)):
        planes, rows, ld = ops.gemm_f32_wide_scratch(m, k)
        assert planes == 3 and ld >= k and (rows == m or rows % 128 == 0)
        assert 6 * rows * ld <= max(ops.F32_PARTS_BYTES, 128 * 6 * ld)


def test_wide_products_refuse_what_they_cannot_cut():
    ops = _ops()
    x, w, out = torch.zeros(70, 64, device=DEV), torch.zeros(8, 64, device=DEV), torch.zeros(70, 8, device=DEV)
    for cut in (dict(tile=24), dict(tile=144), dict(splits=2), dict(splits=3)):
        with pytest.raises(ops.KernelError, match="no tiles"):
            ops.gemm_f32_wide(x, w, out, ops.EPI_STORE_F32, **cut)
    with pytest.raises(ops.KernelError, match="scratch"):
        ops.gemm_f32_wide(x, w, out, ops.EPI_STORE_F32, parts=torch.zeros(3, 70, 32, device=DEV, dtype=torch.bfloat16))
