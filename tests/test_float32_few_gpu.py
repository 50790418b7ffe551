"""Float32 products of a few rows, whose weights pass through a ring per warp, where the ring, the cut of K and the groups of rows
have their edges: against 64 bits, and the same bits on every run."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m, n, k", [
    (4, 8200, 1536),                       # several groups per block, the shorter ring
    (1, 4000, 388), (2, 9000, 132),        # fewer steps in a group than the ring has slots
    (1, 40, 4), (8, 8200, 1040), (16, 5000, 2052),
    (3, 130, 18944), (8, 30, 18944), (16, 40, 18944),      # K over the most blocks; the largest X that fits
    (16, 40, 30000),                       # and one that does not
    # weights in registers, where a ring would leave room for fewer blocks: steps that do not fill the registers, several groups
    (8, 4100, 2052), (16, 3000, 2052), (5, 900, 18948), (4, 620, 40964), (2, 620, 45004), (1, 620, 90004), (8, 70, 40964),
])
def test_few_rows(m, n, k):
    from rust_inference_b200.kernels import ops, tcgen05
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    x = torch.randn(m, k, device=DEV, generator=g)
    w, w2 = (torch.randn(n, k, device=DEV, generator=g) / k ** 0.5 for _ in range(2))
    ref, ref2 = x.double() @ w.double().t(), x.double() @ w2.double().t()
    # a lane's running sum of k / 32 terms, five additions over the lanes and at most eight over blocks: each rounds by 2^-24 of a sum
    # whose size is that of the result, about 1; errors of both signs, the largest of m n a few times their root mean square
    tol = 6 * (k / 32 + 16) ** 0.5 * 2.0 ** -24 * ref.abs().max().item()

    def run(mode, start, **kw):
        out, again = start.clone(), start.clone()
        ops.gemm_f32(x, w, out, mode, **kw)
        ops.gemm_f32(x, w, again, mode, **kw)
        assert torch.equal(out, again)
        return out.double()

    before = torch.randn(m, n, device=DEV, generator=g)
    assert (run(ops.EPI_STORE_F32, before) - ref).abs().max().item() <= tol
    assert (run(ops.EPI_RESIDUAL, before) - (before + ref)).abs().max().item() <= tol + 2.0 ** -22
    want = torch.nn.functional.silu(ref) * ref2
    size = 1 + ref.abs().max().item() + ref2.abs().max().item()
    assert (run(ops.EPI_SILU_MUL, before, w2=w2) - want).abs().max().item() <= tol * size
    torch.cuda.synchronize()
    tcgen05.check_f32_status()
