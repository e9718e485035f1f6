"""The tcgen05 product over inputs larger than a band: rows taken band by band, a last band that is shorter, a row of tiles that is
larger than a band by itself."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("m, n, k", [(2731, 776, 3072), (6000, 264, 3080), (2100, 1600, 8192), (700, 520, 65536)])
def test_products_in_bands(m, n, k):
    a, w = torch.randn(m, k, device=DEV).bfloat16(), torch.randn(n, k, device=DEV).bfloat16()
    out = torch.full((m + 2, n), 7.0, device=DEV)
    kernels.linear_tcgen05(a, w, None, out, m=m)
    want = a.double() @ w.double().t()
    # the products of bfloat16 numbers are exact; the accumulator takes 16 of them at a time and is cut, not rounded, to 24
    # bits: up to one unit in the last place, 2^-23, of a partial sum each time
    assert float((out[:m].double() - want).norm() / want.norm()) < (k / 16 + 2) * 2.0 ** -23
    assert float((out[m:] - 7.0).abs().max()) == 0.0
