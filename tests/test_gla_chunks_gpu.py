"""Long runs of the linear attention with a decay a key channel, whose chunks go to tensor cores in parts: channels in one operand tile and in
several, value channels that leave a block's last columns empty, chunks of one token, decays near one and so strong that no power of
them may be formed alone.  Against the recurrence in 64 bits: the results are those of 32-bit sums and weights."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda", torch.float64


def rel(got, want):
    return float((got.to(F64) - want).norm() / want.norm())


@pytest.mark.parametrize("heads, dim, vdim", [(40, 16, 8), (16, 64, 64), (20, 48, 72), (5, 32, 200), (16, 96, 64)])
@pytest.mark.parametrize("lengths", [[65, 129, 640], [1000, 1, 64, 700]])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("strength", [0.05, 1.0, 30.0])
def test_chunks(heads, dim, vdim, lengths, dtype, strength):
    torch.manual_seed(dim + vdim)
    starts = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    slots = [len(lengths) - i for i in range(len(lengths))]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    n, wide = starts[-1], heads * (2 * dim + vdim)
    proj = torch.randn(n, wide + 8, device=DEV).to(dtype)
    dt = torch.rand(n, heads * dim, device=DEV) * strength
    state = torch.randn(len(lengths) + 1, heads, dim, vdim, device=DEV)
    first, out = state.clone(), torch.full((n, heads * vdim), 7.0, device=DEV)
    scratch = torch.full((kernels.gla_chunked_scratch_floats(n, len(lengths), max(lengths), heads, dim, vdim),), float("nan"), device=DEV)
    kernels.gla_scan(proj, 0, heads * dim, 2 * heads * dim, dim ** -0.5, dt, -0.25, state, ints(slots), ints(starts), out,
                     n_seqs=len(lengths), n_heads=heads, dim=dim, vdim=vdim, max_new=max(lengths), scratch=scratch)
    x = proj.to(F64)
    for i, (lo, hi) in enumerate(zip(starts[:-1], starts[1:])):
        q, k, v = (x[lo:hi, a:b].reshape(hi - lo, heads, -1) for a, b in
                   ((0, heads * dim), (heads * dim, 2 * heads * dim), (2 * heads * dim, wide)))
        decay = torch.exp(-0.25 * dt[lo:hi].to(F64)).view(hi - lo, heads, dim)
        S, want = first[slots[i]].to(F64), []
        for t in range(hi - lo):
            S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            want.append(torch.einsum("hkv,hk->hv", S, q[t] * dim ** -0.5).reshape(-1))
        # a weight is e to a 32-bit sum of up to 64 log decays that are themselves up to 7.5 each
        assert rel(out[lo:hi], torch.stack(want)) < 1e-6 and rel(state[slots[i]], S) < 1e-6
    assert torch.equal(state[0], first[0])
