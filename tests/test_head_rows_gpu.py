"""One product of all heads' weights whose columns go to the heads' own places, against float64: heads of one and several pieces of
32, rows past a tile's edge, rows and heads apart, what lies between them left alone."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("tokens", [65, 128, 257, 700])
@pytest.mark.parametrize("heads, n, beside, k", [(3, 32, 8, 72), (5, 64, 64, 512), (2, 96, 16, 256), (12, 64, 0, 264)])
def test_rows_of_heads(tokens, heads, n, beside, k):
    a = torch.randn(tokens, k + 24, device=DEV).bfloat16()[:, :k]
    w = torch.randn(heads * n, k, device=DEV).bfloat16()
    store = torch.full((heads, tokens, n + beside), 7.0, device=DEV).bfloat16()
    out = store.transpose(0, 1)[:, :, :n]
    assert kernels.head_rows_supports(a, w, out, tokens)
    kernels.head_rows(a, w, out, n_tokens=tokens)
    want = (a.double() @ w.double().t()).view(tokens, heads, n)
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -8      # (one rounding to 8 bits)
    assert bool((store[:, :, n:] == 7.0).all())


def test_what_it_does_not_take():
    a, w = torch.randn(100, 64, device=DEV).bfloat16(), torch.randn(80, 64, device=DEV).bfloat16()
    out = torch.empty(2, 100, 40, device=DEV, dtype=torch.bfloat16).transpose(0, 1)
    assert not kernels.head_rows_supports(a, w, out, 100)                     # heads of 40
    out = torch.empty(2, 100, 64, device=DEV, dtype=torch.bfloat16).transpose(0, 1)
    w = torch.randn(128, 64, device=DEV).bfloat16()
    assert kernels.head_rows_supports(a, w, out, 100) and not kernels.head_rows_supports(a, w, out, 64)
