"""The experts' lists, at the sizes where the arranging block's parts change: pairs beyond those it holds in registers, experts beyond a
warp's lanes, ids that name no expert, rows gathered with the lists."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("tokens, top, experts, rows, stray", [(1, 1, 1, 128, 0), (8, 4, 32, 128, 0), (64, 4, 33, 16, 0), (50, 5, 100, 128, 3),
                                                               (2048, 4, 32, 128, 0), (2049, 4, 64, 128, 0), (3000, 7, 257, 32, 9)])
def test_lists_of_the_experts(tokens, top, experts, rows, stray):
    from rust_inference_b200.kernels import ops
    pairs = tokens * top
    i32 = lambda n: torch.full((n,), -7, dtype=torch.int32, device=DEV)
    ids = torch.randint(0, experts + stray, (tokens, top), dtype=torch.int32, device=DEV)
    offsets, order, tiles, n_tiles, place = i32(experts + 1), i32(pairs), i32(2 * (-(-pairs // rows) + experts)), i32(1), i32(pairs)
    gather = pairs <= 256
    x = torch.randn(tokens, 64, device=DEV).bfloat16()
    xs = torch.zeros(pairs, 64, device=DEV, dtype=torch.bfloat16)
    ops.moe_arrange(ids, pairs, experts, rows, offsets, order, tiles, n_tiles, place, gather=(x, xs, top) if gather else None)
    flat, got = ids.view(-1).cpu().tolist(), order.cpu().tolist()
    want = [[p for p, e in enumerate(flat) if e == k] for k in range(experts)]
    starts = offsets.cpu().tolist()
    assert starts == [sum(len(v) for v in want[:k]) for k in range(experts + 1)]
    assert all(sorted(got[starts[k]:starts[k + 1]]) == want[k] for k in range(experts))
    places = place.cpu().tolist()
    assert all(places[p] == at for at, p in enumerate(got[:starts[-1]]))
    assert tiles.cpu()[:2 * int(n_tiles)].view(-1, 2).tolist() == [[k, starts[k] + r] for k in range(experts) for r in range(0, len(want[k]), rows)]
    if gather:
        assert torch.equal(xs[:starts[-1]], x[order[:starts[-1]].long() // top])
