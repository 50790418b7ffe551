"""The recurrences' pieces with two and four value columns per thread, against the same tokens in one pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("lengths, heads, dim, vdim", [([1300], 8, 128, 128), ([200, 1, 513, 64], 16, 100, 72), ([400, 130], 20, 24, 130),
                                                       ([300], 2, 128, 128), ([257], 3, 250, 65),
                                                       # blocks of two columns that just fit the SMs together, and that do not
                                                       ([770], 16, 64, 128), ([900], 16, 64, 128), ([1180], 8, 128, 128)])
def test_pieces_are_the_one_pass(lengths, heads, dim, vdim):
    from rust_inference_b200.kernels import ops
    n, b, piece = sum(lengths), len(lengths), 64
    most = -(-max(lengths) // piece)
    cu = _i32([sum(lengths[:i]) for i in range(b + 1)])
    slot = _i32(list(range(b, 0, -1)))
    z0 = torch.randn(n, 2 * heads * dim + heads * vdim, device=DEV)
    bias, low = torch.randn(heads * dim, device=DEV), torch.rand(heads * dim, device=DEV) * 0.9
    state0 = torch.randn(b + 1, heads, dim, vdim, device=DEV)
    got = {}
    for p in (0, piece):
        state, out, raw = state0.clone(), torch.empty(n, heads * vdim, device=DEV), torch.empty(n, heads * vdim, device=DEV)
        scratch = torch.empty(b * most * heads * dim * (vdim + 1), device=DEV)
        ops.gated_recurrence(z0.clone(), bias, low, torch.ones(vdim, device=DEV), state, cu, slot, out, n_seqs=b, heads=heads, dim=dim,
                             vdim=vdim, eps=1e-5, o_raw=raw, piece=p, max_pieces=most if p else 1, scratch=scratch if p else None,
                             longest_run=max(lengths))
        got[p] = out, raw, state
    # a piece's start state takes one rounding of its own per piece in place of one per token
    for one, cut in zip(got[0], got[piece]):
        assert float((one - cut).norm() / one.norm()) <= 64 * 2.0 ** -24
    assert torch.equal(got[0][2][0], state0[0]) and torch.equal(got[piece][2][0], state0[0])      # the slot nobody has
