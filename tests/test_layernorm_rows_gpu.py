"""LayerNorm of many rows: both sides of the number of rows up to which its weights are read early, odd numbers of rows, every number of
vectors a lane holds; rows picked by an index.  Against 64 bits, and a row alone against the same row among all."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [64, 4095, 4096, 4097, 9001])
@pytest.mark.parametrize("width", [768, 1280, 1600, 2048])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_many_rows(n, width, out_dtype):
    torch.manual_seed(n + width)
    x, g, b = torch.randn(n, width, device=DEV) * 5.0 + 100.0, torch.randn(width, device=DEV), torch.randn(width, device=DEV)
    out = torch.full((n + 1, width), 7.0, device=DEV).to(out_dtype)
    kernels.layernorm(x, g, b, out, 1e-5, n_rows=n)
    want = torch.nn.functional.layer_norm(x.double(), (width,), g.double(), b.double(), 1e-5)
    # a mean of 100 beside a spread of 5: 32-bit differences of 2^-24 of 100 relative to 5; bfloat16 rounds once
    assert float((out[:n].double() - want).norm() / want.norm()) < (5e-6 if out_dtype is torch.float32 else 2.0 ** -8.5)
    assert bool((out[n] == 7.0).all())
    alone = torch.empty(1, width, device=DEV, dtype=out_dtype)
    kernels.layernorm(x[n - 1:], g, b, alone, 1e-5)
    assert torch.equal(alone[0], out[n - 1])
    rows = torch.randperm(n, device=DEV).to(torch.int32)
    picked = torch.empty(n, width, device=DEV, dtype=out_dtype)
    kernels.layernorm(x, g, b, picked, 1e-5, rows=rows)
    assert torch.equal(picked, out[:n][rows.long()])
