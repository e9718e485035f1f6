"""The matrix memory's normaliser over long runs, whose weights are exactly one here: what is left of an error is that of its sums."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda", torch.float64


@pytest.mark.parametrize("dim", [16, 48, 64, 128])
def test_sums_are_rounded_and_not_cut(dim):
    torch.manual_seed(dim)
    heads, vdim, n = 64, 16, 128
    wide = heads * (2 * dim + vdim)
    proj = torch.zeros(n, wide + 2 * heads, device=DEV)
    proj[:, wide + heads:] = 190.0      # a log forget gate of zero, as the input gate's; maxima stay at zero
    proj[:, heads * dim:2 * heads * dim] = torch.rand(n, heads * dim, device=DEV) + 0.5
    s, norm, m = (torch.zeros(1, heads, *d, device=DEV) for d in ((dim, vdim), (dim,), ()))
    none, out = torch.zeros(heads, device=DEV), torch.empty(n, heads * vdim, device=DEV)
    scratch = torch.empty(kernels.mlstm_chunked_scratch_floats(n, 1, n, heads, dim, vdim), device=DEV)
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    kernels.mlstm_scan(proj, (0, heads * dim, 2 * heads * dim, wide, wide + heads), none, none, 200.0, 1.0, s, norm, m, ints(0), ints(0, n),
                       out, n_seqs=1, n_heads=heads, dim=dim, vdim=vdim, max_new=n, scratch=scratch)
    want = proj[:, heads * dim:2 * heads * dim].to(F64).sum(0).view(1, heads, dim)
    error = (norm.to(F64) - want) / want
    # sums of 64 numbers rounded as often: up to 1e-7 each in the norm, without a sign, so that a thousand and more of them average out
    assert float(error.pow(2).mean().sqrt()) < 1e-7 and abs(float(error.mean())) < 2e-8


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_read_out_with_one_large_channel(dim, dtype):
    torch.manual_seed(dim)
    heads, vdim, n = 64, 16, 128
    wide = heads * (2 * dim + vdim)
    proj = torch.zeros(n, wide + 2 * heads, device=DEV)
    proj[:, wide + heads:] = 190.0
    q = torch.rand(n, heads, dim, device=DEV) + 0.5
    q[:, :, 0] = 1.0
    proj[:, :heads * dim] = q.view(n, -1)
    proj = proj.to(dtype)
    norm, m = torch.rand(1, heads, dim, device=DEV) + 0.5, torch.zeros(1, heads, device=DEV)
    norm[:, :, 0] = 4096.0 * (1.0 + torch.rand(1, heads, device=DEV))
    s = torch.zeros(1, heads, dim, vdim, device=DEV)
    s[:, :, 0] = 2.0 ** 20      # what is divided is exact
    den = torch.einsum("thd,hd->th", proj[:, :heads * dim].to(F64).view(n, heads, dim), norm[0].to(F64))
    none, out = torch.zeros(heads, device=DEV), torch.empty(n, heads * vdim, device=DEV)
    scratch = torch.empty(kernels.mlstm_chunked_scratch_floats(n, 1, n, heads, dim, vdim), device=DEV)
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    kernels.mlstm_scan(proj, (0, heads * dim, 2 * heads * dim, wide, wide + heads), none, none, 200.0, 1.0, s, norm, m, ints(0), ints(0, n),
                       out, n_seqs=1, n_heads=heads, dim=dim, vdim=vdim, max_new=n, scratch=scratch)
    error = out.to(F64).view(n, heads, vdim)[:, :, 0] * (den + 1e-6) / 2.0 ** 20 - 1.0
    # the sum of the large channel's 16 is cut once (2^-23 at most), the up to seven others are added with a rounding each (2^-24, no sign)
    assert float(error.pow(2).mean().sqrt()) < 2e-7
