"""The router's kernel for rows of whole pieces, a token or four a block, and the sorting of pairs beyond what its threads hold."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("experts,k,top", [(3, 8, 2), (9, 1016, 3), (16, 24, 4), (32, 512, 4), (33, 256, 8), (64, 1016, 8), (1024, 64, 32)])
def test_a_token_alone_and_among_others(dtype, experts, k, top):
    if dtype == torch.float32:
        k //= 2
    torch.manual_seed(experts)
    n = 1001
    x, router = (torch.randn(r, k, device=DEV).to(dtype) for r in (n, experts))
    bias = torch.randn(experts, device=DEV) * 0.1
    ids, weights = torch.empty(n, top, dtype=torch.int32, device=DEV), torch.empty(n, top, device=DEV)
    kernels.moe_route(x, router, ids, weights, n_tokens=n, top=top, choice_bias=bias)
    for first, count in ((0, 1), (500, 2), (998, 3), (100, 290)):
        few_ids, few = torch.empty(count, top, dtype=torch.int32, device=DEV), torch.empty(count, top, device=DEV)
        kernels.moe_route(x[first:first + count], router, few_ids, few, n_tokens=count, top=top, choice_bias=bias)
        assert torch.equal(few_ids, ids[first:first + count]) and torch.equal(few, weights[first:first + count])
    # against 64 bits: k products a sum (roundings of 2^-24 each, a few of which meet), and a sigmoid
    score = torch.sigmoid(x.double() @ router.double().T)
    chosen = (score + bias.double()).topk(top).values
    mine = torch.gather(score + bias.double(), 1, ids.long())
    assert float((mine - chosen).abs().max()) < 1e-5
    picked = torch.gather(score, 1, ids.long())
    torch.testing.assert_close(weights.double(), picked / picked.sum(1, keepdim=True), rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("pairs,experts", [(1, 1), (100, 70), (16384, 64), (16385, 3), (40000, 200)])
def test_sort(pairs, experts):
    torch.manual_seed(pairs)
    ids = torch.randint(0, experts, (pairs,), dtype=torch.int32, device=DEV)
    offsets, tiles = (torch.empty(experts + 1, dtype=torch.int32, device=DEV) for _ in range(2))
    order, place = (torch.full((pairs,), -1, dtype=torch.int32, device=DEV) for _ in range(2))
    kernels.moe_sort(ids, offsets, tiles, order, place, pairs=pairs, n_experts=experts)
    counts = torch.bincount(ids.long(), minlength=experts)
    assert torch.equal(offsets[1:].long(), counts.cumsum(0)) and int(offsets[0]) == 0 and int(tiles[0]) == 0
    rows = kernels.library().bt_moe_tile_rows()
    assert torch.equal(tiles[1:].long(), ((counts + rows - 1) // rows).cumsum(0))
    assert torch.equal(order[place.long()].long(), torch.arange(pairs, device=DEV))
    assert torch.equal(ids[order.long()], ids.sort().values)
