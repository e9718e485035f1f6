"""The routed experts' products on tcgen05: experts with no row, with one, with whole tiles and with one more; columns and K that
end inside a tile; rows of experts without tensors behind the others'."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("counts, behind", [([128, 0, 1, 129, 300, 256], 0), ([0, 0, 500], 37), ([640], 0), ([3] * 70 + [200], 5)])
@pytest.mark.parametrize("width, inner", [(128, 64), (264, 136), (96, 40), (1024, 512)])
@pytest.mark.parametrize("mode", ["pair", "plain"])
def test_experts_products(counts, behind, width, inner, mode):
    experts, top, pairs = len(counts), 2, sum(counts) + behind
    pairs += pairs % 2
    tokens = pairs // top
    gen = torch.Generator(device=DEV).manual_seed(3)
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)] + [torch.full((pairs - sum(counts),), experts)])
    ids = ids[torch.randperm(pairs)].to(torch.int32).to(DEV)
    routes = experts + 1
    offsets, tile_first = (torch.empty(routes + 1, dtype=torch.int32, device=DEV) for _ in range(2))
    order, place = (torch.empty(pairs, dtype=torch.int32, device=DEV) for _ in range(2))
    kernels.moe_sort(ids, offsets, tile_first, order, place, pairs=pairs, n_experts=routes)
    rand = lambda *s, std=1.0: torch.randn(s, generator=gen, device=DEV) * std  # noqa: E731
    x = rand(tokens, width).bfloat16()
    halves = 2 if mode == "pair" else 1
    w_in, w_out = rand(experts, halves * inner, width, std=width ** -0.5).bfloat16(), rand(experts, width, inner, std=inner ** -0.5).bfloat16()
    weights = torch.rand(pairs, generator=gen, device=DEV)
    rows = torch.empty(pairs, width, dtype=torch.bfloat16, device=DEV)
    kernels.moe_gather(x, order, rows, pairs=pairs, top=top)
    assert torch.equal(rows, x[(order // top).long()])
    hidden = torch.full((pairs, inner), 7.0, device=DEV).bfloat16()
    kernels.moe_expert_tcgen05(True, rows, w_in, hidden, offsets, order, None, pairs=pairs, gated=mode == "pair",
                               activation="swish" if mode == "pair" else "gelu_new")
    part = torch.full((pairs, width), 7.0, device=DEV)
    kernels.moe_expert_tcgen05(False, hidden, w_out, part, offsets, order, weights, pairs=pairs)
    at = 0
    for e, c in enumerate(counts):
        if c == 0:
            continue
        z = rows[at:at + c].double() @ w_in[e].double().t()
        want = torch.nn.functional.silu(z[:, :inner]) * z[:, inner:] if mode == "pair" else torch.nn.functional.gelu(z, approximate="tanh")
        assert rel(hidden[at:at + c], want) < 2.0 ** -8            # (one rounding to 8 bits)
        want = hidden[at:at + c].double() @ w_out[e].double().t() * weights[order[at:at + c].long()].double()[:, None]
        # (exact products; the accumulator is cut to 24 bits once for 16 of them)
        assert rel(part[at:at + c], want) < (inner / 16 + 2) * 2.0 ** -23
        at += c
    assert bool((part[at:] == 7.0).all()) and bool((hidden[at:] == 7.0).all())
    kernels.check_status(x.device)
