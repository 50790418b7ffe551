"""The gated product of a few tokens whose K is cut over the blocks of a cluster, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m", [1, 2, 3, 7, 8, 9, 16])
@pytest.mark.parametrize("n, k", [(128, 512), (391, 192), (1000, 2056)])
@pytest.mark.parametrize("cluster", [1, 2, 3, 8])
def test_gated_product_cut_over_a_cluster(m, n, k, cluster):
    from rust_inference_b200.kernels import linear, ops, tcgen05
    cluster = min(cluster, -(-k // 64))
    x = (torch.randn(m, k, device=DEV) * 0.5).bfloat16()
    w, w2 = (linear.Weight((torch.randn(n, k, device=DEV) * 0.1).bfloat16()) for _ in range(2))
    gate, up = (x.double() @ t.t.double().t() for t in (w, w2))
    want = gate * torch.sigmoid(gate) * up
    out = torch.full((m, n), 9.0, device=DEV, dtype=torch.bfloat16)
    tcgen05.gemm(x, w, out, ops.EPI_SILU_MUL, w2=w2, split_k=cluster)
    # one rounding to bfloat16 (2^-9) of each result, and float32 sums of k products (k * 2^-24 of their size)
    assert float(((out.double() - want).norm() / want.norm())) <= 2.0 ** -8
    torch.cuda.synchronize()
    tcgen05.check_status()


def test_gated_product_refuses_clusters_it_cannot_form():
    from rust_inference_b200.kernels import linear, ops, tcgen05
    w = linear.Weight(torch.zeros(128, 1024, device=DEV, dtype=torch.bfloat16))
    for m, cluster in ((17, 2), (200, 2), (4, 9)):
        x = torch.zeros(m, 1024, device=DEV, dtype=torch.bfloat16)
        with pytest.raises(ops.KernelError, match="no cluster"):
            tcgen05.gemm(x, w, torch.zeros(m, 128, device=DEV, dtype=torch.bfloat16), ops.EPI_SILU_MUL, w2=w, split_k=cluster)


@pytest.mark.parametrize("m", [1, 5, 16])
@pytest.mark.parametrize("n, k, cluster", [(128, 512, 2), (391, 1000, 3), (72, 2056, 8), (1000, 640, 4)])
def test_plain_products_cut_over_a_cluster(m, n, k, cluster):
    from rust_inference_b200.kernels import linear, ops, tcgen05
    x = (torch.randn(m, k, device=DEV) * 0.5).bfloat16()
    w = linear.Weight((torch.randn(n, k, device=DEV) * 0.1).bfloat16())
    bias, cols = torch.randn(n, device=DEV), torch.tensor([n // 2], dtype=torch.float32, device=DEV)
    ref = x.double() @ w.t.double().t()
    out32, part = torch.full((m, n), 9.0, device=DEV), torch.full((m, n), 9.0, device=DEV)
    out = torch.full((m, n), 9.0, device=DEV, dtype=torch.bfloat16)
    tcgen05.gemm(x, w, out32, ops.EPI_STORE_F32, split_k=cluster)
    tcgen05.gemm(x, w, out, ops.EPI_STORE, bias=bias, split_k=cluster)
    tcgen05.gemm(x, w, part, ops.EPI_SILU_F32, silu_cols=cols, split_k=cluster)
    # float32 sums of k products; one rounding to bfloat16; the quick exponential and division of the activated columns
    assert float((out32.double() - ref).norm() / ref.norm()) <= 1e-5
    assert float((out.double() - ref - bias).norm() / (ref + bias).norm()) <= 2.0 ** -8
    want = torch.cat([ref[:, :n // 2] * torch.sigmoid(ref[:, :n // 2]), ref[:, n // 2:]], dim=1)
    assert float((part.double() - want).norm() / want.norm()) <= 1e-5
    torch.cuda.synchronize()
    tcgen05.check_status()


@pytest.mark.parametrize("m", [1, 8, 9, 12, 16, 17])
@pytest.mark.parametrize("n, k, cluster", [
    (4096, 1032, 4), (4736, 1024, 4),                # 32 tiles, and 37: more clusters of four than SMs hold one by one
    (5120, 1024, 3), (6144, 1024, 3),                # 40 tiles, and 48: the same for clusters of three
    (8960, 640, 2), (18944, 512, 1), (1024, 448, 1)])
def test_planned_clusters(n, k, cluster, m):
    """The plan's own cut, whose sums are the same on every run and those of the cut asked for by number."""
    from rust_inference_b200.kernels import linear, ops, tcgen05
    x = (torch.randn(m, k, device=DEV) * 0.5).bfloat16()
    w, w2 = (linear.Weight((torch.randn(n, k, device=DEV) * 0.1).bfloat16()) for _ in range(2))
    cluster = 1 if m > 16 else cluster
    ref, up = (x.double() @ t.t.double().t() for t in (w, w2))
    # gated: one rounding to bfloat16; stored: float32 sums of k products
    for mode, extra, want, tol in ((ops.EPI_SILU_MUL, dict(w2=w2), ref * torch.sigmoid(ref) * up, 2.0 ** -8), (ops.EPI_STORE_F32, {}, ref, 1e-5)):
        assert tcgen05.plan(m, n, k, mode)[1] == cluster
        out = torch.full((m, n), 9.0, device=DEV, dtype=torch.bfloat16 if extra else torch.float32)
        again, asked = out.clone(), out.clone()
        tcgen05.gemm(x, w, out, mode, **extra)
        tcgen05.gemm(x, w, again, mode, **extra)
        tcgen05.gemm(x, w, asked, mode, split_k=cluster, **extra)
        assert torch.equal(out, again) and torch.equal(out, asked)
        assert float((out.double() - want).norm() / want.norm()) <= tol
    torch.cuda.synchronize()
    tcgen05.check_status()
