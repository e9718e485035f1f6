"""The tcgen05 product on pairs of blocks: rows that leave a pair's second block empty, partly or wholly filled, columns and K
that end inside a tile, one tile and several a pair."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("m, n, k", [(129, 64, 4096), (255, 768, 3072), (256, 776, 3080), (257, 768, 3072), (385, 1600, 1000),
                                     (1025, 1016, 4096), (2048, 768, 3072), (2049, 1024, 2816), (4100, 1600, 640),
                                     (9000, 1608, 328)])
def test_products_of_pairs(m, n, k):
    a, w = torch.randn(m, k, device=DEV).bfloat16(), torch.randn(n, k, device=DEV).bfloat16()
    bias, res = torch.randn(n, device=DEV), torch.randn(m, n, device=DEV)
    want = a.double() @ w.double().t() + bias.double()
    out = torch.cat([res, torch.full((2, n), 7.0, device=DEV)])
    kernels.linear_tcgen05(a, w, bias, out, m=m, residual=out)
    # the products of bfloat16 numbers are exact; the accumulator takes 16 of them at a time and is cut, not rounded, to 24
    # bits: up to one unit in the last place, 2^-23, of a partial sum each time
    assert rel(out[:m], want + res.double()) < (k / 16 + 2) * 2.0 ** -23
    assert float((out[m:] - 7.0).abs().max()) == 0.0
    low = torch.empty(m, n, device=DEV, dtype=torch.bfloat16)
    kernels.linear_tcgen05(a, w, bias, low, m=m)
    assert rel(low, want) < 2.0 ** -8            # (one rounding to 8 bits)


def test_a_row_does_not_depend_on_how_its_tile_is_cut():
    a, w = torch.randn(2048, 3072, device=DEV).bfloat16(), torch.randn(768, 3072, device=DEV).bfloat16()
    whole, part = torch.empty(2048, 768, device=DEV), torch.empty(70, 768, device=DEV)
    kernels.linear_tcgen05(a, w, None, whole, m=2048)
    kernels.linear_tcgen05(a[1000:1070].contiguous(), w, None, part, m=70)
    assert torch.equal(whole[1000:1070], part)
