"""The recurrences' chunks on tensor cores at the ends of the numbers' range: x sigmoid(x) far below zero."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda", torch.float64


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_feature_far_below_zero(dtype):
    heads, dim, n = 16, 16, 640
    values = torch.tensor([-20.0, -60.0, -86.5, -87.5, -88.5, -95.0, -104.0, -1e10, -1e30, -3e38], device=DEV).to(dtype)
    proj = torch.full((n, 3 * heads * dim), 1e4, device=DEV, dtype=dtype)
    proj[:, 2 * heads * dim:] = values.repeat(n * heads * dim // len(values)).view(n, -1)
    state, out = torch.zeros(1, heads, dim, dim, device=DEV), torch.empty(n, heads * dim, device=DEV)
    scratch = torch.empty(kernels.lightning_chunked_scratch_floats(1, n, heads, dim, dim), device=DEV)
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    kernels.lightning_scan(proj, 0, heads * dim, 2 * heads * dim, state, ints(0), ints(0, n), torch.zeros(heads, device=DEV), out, n_seqs=1,
                           n_heads=heads, dim=dim, vdim=dim, max_new=n, scratch=scratch)
    v = proj[:, 2 * heads * dim:].to(F64)
    want = dim * proj[0, 0].to(F64) ** 2 * v / (1.0 + torch.exp(-v))      # (a decay of zero: a token sees itself alone)
    # (below 2^-110 a number's parts have fewer bits: the last of bfloat16's numbers is 2^-133)
    error = float(((out.to(F64) - want).abs() / (1e-5 * want.abs() + dim * 1e8 * 2.0 ** -132)).max())
    assert error < 1.0
