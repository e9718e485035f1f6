"""Long runs of the recurrences alone and among others: a sequence's results and state are the same bits in each call."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


def ints(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("heads, dim, vdim", [(4, 64, 64), (3, 128, 96), (4, 16, 24)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("activation", ["swish", None])
def test_decayed(heads, dim, vdim, dtype, activation):
    torch.manual_seed(dim)
    proj, wide = torch.randn(200 * 16, heads * (2 * dim + vdim), device=DEV).to(dtype), heads * dim
    decay, first = torch.rand(heads, device=DEV) * 0.6 + 0.4, torch.randn(1, heads, dim, vdim, device=DEV)
    seen = []
    for lengths in ([200], [200] * 16, [200, 3000]):
        n, k = sum(lengths), len(lengths)
        state, out = first.repeat(k, 1, 1, 1), torch.empty(n, heads * vdim, device=DEV)
        scratch = torch.empty(kernels.lightning_chunked_scratch_floats(k, max(lengths), heads, dim, vdim), device=DEV)
        kernels.lightning_scan(proj[:n], 0, wide, 2 * wide, state, ints(range(k)), ints([sum(lengths[:i]) for i in range(k + 1)]), decay, out,
                               n_seqs=k, n_heads=heads, dim=dim, vdim=vdim, max_new=max(lengths), scratch=scratch, activation=activation)
        seen.append((out[:200], state[0]))
    assert all(torch.equal(a, b) for other in seen[1:] for a, b in zip(seen[0], other))


@pytest.mark.parametrize("heads, dim, vdim", [(4, 64, 64), (3, 128, 96), (4, 16, 24)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_memory(heads, dim, vdim, dtype):
    torch.manual_seed(dim)
    wide = heads * (2 * dim + vdim)
    proj = torch.randn(200 * 16, wide + 2 * heads, device=DEV).to(dtype)
    bias_i, bias_f = torch.randn(heads, device=DEV) - 1.0, torch.rand(heads, device=DEV) * 4.0 + 1.0
    first = [torch.randn(1, heads, *d, device=DEV) for d in ((dim, vdim), (dim,), ())]
    seen = []
    for lengths in ([200], [200] * 16, [200, 3000]):
        n, k = sum(lengths), len(lengths)
        s, nn, m = (t.repeat(k, *(1,) * (t.dim() - 1)) for t in first)
        out = torch.empty(n, heads * vdim, device=DEV)
        scratch = torch.empty(kernels.mlstm_chunked_scratch_floats(n, k, max(lengths), heads, dim, vdim), device=DEV)
        kernels.mlstm_scan(proj[:n], (0, heads * dim, 2 * heads * dim, wide, wide + heads), bias_i, bias_f, 15.0, dim ** -0.5, s, nn, m,
                           ints(range(k)), ints([sum(lengths[:i]) for i in range(k + 1)]), out, n_seqs=k, n_heads=heads, dim=dim, vdim=vdim,
                           max_new=max(lengths), scratch=scratch)
        seen.append((out[:200], s[0], nn[0], m[0]))
    assert all(torch.equal(a, b) for other in seen[1:] for a, b in zip(seen[0], other))
