"""The routed experts' products below the tcgen05 products' sizes: more of K than a turn of the loop takes, rows that fill one row
tile and two, each side of the kernels' rule; and rows and weights that the tcgen05 products do not take."""
import types

import pytest
import torch

from burn_transformers_b200 import kernels
from burn_transformers_b200.parts.routed import RoutedFeedForward

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


# (16 rows an expert on average and fewer stream the weights; many experts at 17 and more, and few at 100, stage both operands)
@pytest.mark.parametrize("counts", [[1, 0, 16, 3], [31, 32, 33, 48], [0, 96, 0, 0], [200, 100, 64, 65], [17] * 130, [2] * 300])
@pytest.mark.parametrize("width, inner", [(40, 24), (264, 520), (512, 136), (1032, 72)])
@pytest.mark.parametrize("gated", [True, False])
def test_products_of_few_rows(counts, width, inner, gated):
    experts, top, pairs = len(counts), 2, sum(counts)
    gen = torch.Generator(device=DEV).manual_seed(3)
    rand = lambda *s, std=1.0: torch.randn(s, generator=gen, device=DEV) * std  # noqa: E731
    ids = torch.cat([torch.full((c,), e) for e, c in enumerate(counts)])[torch.randperm(pairs)].to(torch.int32).to(DEV)
    offsets, tile_first = (torch.empty(experts + 1, dtype=torch.int32, device=DEV) for _ in range(2))
    order, place = (torch.empty(pairs, dtype=torch.int32, device=DEV) for _ in range(2))
    kernels.moe_sort(ids, offsets, tile_first, order, place, pairs=pairs, n_experts=experts)
    x = rand(-(-pairs // top), width).bfloat16()
    w_in = rand(experts, (2 if gated else 1) * inner, width, std=width ** -0.5).bfloat16()
    w_out, weights = rand(experts, width, inner, std=inner ** -0.5).bfloat16(), torch.rand(pairs, generator=gen, device=DEV)
    hidden, part = torch.empty(pairs, inner, device=DEV, dtype=torch.bfloat16), torch.empty(pairs, width, device=DEV)
    kernels.moe_expert(True, x, w_in, hidden, offsets, tile_first, order, None, pairs=pairs, top=top, gated=gated,
                       activation="swish" if gated else "gelu_new")
    kernels.moe_expert(False, hidden, w_out, part, offsets, tile_first, order, weights, pairs=pairs, top=top)
    of = torch.repeat_interleave(torch.arange(experts, device=DEV), torch.tensor(counts, device=DEV))      # (each sorted row's expert)
    z = torch.cat([x[(order[of == e] // top).long()].double() @ w_in[e].double().t() for e in range(experts)])
    want = torch.nn.functional.silu(z[:, :inner]) * z[:, inner:] if gated else torch.nn.functional.gelu(z, approximate="tanh")
    assert rel(hidden, want) < 2.0 ** -8            # (one rounding to 8 bits)
    want = torch.cat([hidden[of == e].double() @ w_out[e].double().t() for e in range(experts)]) * weights[order.long()].double()[:, None]
    # (exact products; the accumulator is cut to 24 bits once for 16 of them, the warps' eight sums are rounded)
    assert rel(part, want) < (inner / 16 + 10) * 2.0 ** -23


def test_what_the_tcgen05_products_do_not_take_goes_on():
    """Weights off a 16-byte boundary: as before there were tcgen05 products, another kernel takes them."""
    width, inner, experts, tokens, top = 256, 128, 16, 2048, 2
    gen = torch.Generator(device=DEV).manual_seed(4)
    flat = lambda n, off: (torch.randn(n + off, generator=gen, device=DEV) * 0.06).bfloat16()[off:]  # noqa: E731
    x = torch.randn(tokens, width, generator=gen, device=DEV).bfloat16()
    numbers = flat(experts * 2 * inner * width, 0), flat(experts * width * inner, 0)
    router = torch.randn(experts, width, generator=gen, device=DEV).bfloat16()
    results = []
    for shift in (0, 1):
        part = RoutedFeedForward(width, experts, top, inner, activation="swish")
        w_in, w_out = (torch.empty(w.numel() + shift, dtype=w.dtype, device=DEV)[shift:].copy_(w) for w in numbers)
        part.bind({"router.weight": router, "in.weight": w_in.view(-1, width), "out.weight": w_out.view(-1, inner)})
        assert kernels.moe_many_rows_supports(x, part.w_in, part.w_out, pairs=tokens * top) == (shift == 0)
        ws = types.SimpleNamespace(take=lambda shape, dtype: torch.empty(shape, dtype=dtype, device=DEV), mark=lambda: 0, release=lambda m: None)
        ctx = types.SimpleNamespace(n_tokens=tokens, dtype=torch.bfloat16, ws=ws)
        out = torch.zeros(tokens, width, device=DEV)
        part.forward(ctx, x, out)
        results.append(out)
    # (the experts' inner numbers are rounded to 8 bits, in a few places the other way)
    assert rel(results[1], results[0].double()) < 2.0 ** -8
