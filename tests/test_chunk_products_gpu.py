"""Long runs of the decayed linear attention and of the matrix memory whose chunks go to tensor cores in parts: channels in one operand
tile and in several, value channels that leave a block's last columns empty, chunks of one token, every form of the rows.  Against
the recurrences in 64 bits: the results are those of 32-bit sums."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda", torch.float64


def rel(got, want):
    return float((got.to(F64) - want).norm() / want.norm())


def step(lengths):
    starts = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    slots = [len(lengths) - i for i in range(len(lengths))]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    return starts, slots, ints(starts), ints(slots)


@pytest.mark.parametrize("heads, dim, vdim", [(40, 16, 8), (16, 64, 64), (20, 48, 72), (5, 128, 200), (16, 96, 64)])
@pytest.mark.parametrize("lengths", [[65, 129, 640], [1000, 1, 64, 700]])
@pytest.mark.parametrize("dtype, activation", [(torch.bfloat16, "swish"), (torch.bfloat16, None), (torch.float32, "swish"), (torch.float32, None)])
def test_decayed_chunks(heads, dim, vdim, lengths, dtype, activation):
    torch.manual_seed(dim + vdim)
    starts, slots, seq_start, slot_ids = step(lengths)
    n, wide = starts[-1], heads * (2 * dim + vdim)
    proj = torch.randn(n, wide + 8, device=DEV).to(dtype)
    decay = torch.rand(heads, device=DEV) * 0.6 + 0.4
    state = torch.randn(len(lengths) + 1, heads, dim, vdim, device=DEV)
    first, out = state.clone(), torch.full((n + 2, heads * vdim), 7.0, device=DEV)
    scratch = torch.full((kernels.lightning_chunked_scratch_floats(len(lengths), max(lengths), heads, dim, vdim),), float("nan"), device=DEV)
    kernels.lightning_scan(proj, 0, heads * dim, 2 * heads * dim, state, slot_ids, seq_start, decay, out, n_seqs=len(lengths),
                           n_heads=heads, dim=dim, vdim=vdim, max_new=max(lengths), scratch=scratch, activation=activation)
    x = proj.to(F64)
    x = x * torch.sigmoid(x) if activation else x
    for i, (lo, hi) in enumerate(zip(starts[:-1], starts[1:])):
        q, k, v = (x[lo:hi, a:b].reshape(hi - lo, heads, -1) for a, b in
                   ((0, heads * dim), (heads * dim, 2 * heads * dim), (2 * heads * dim, wide)))
        S, want = first[slots[i]].to(F64), []
        for t in range(hi - lo):
            S = decay.to(F64)[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
            want.append(torch.einsum("hkv,hk->hv", S, q[t]).reshape(-1))
        # sums of some hundred 32-bit products, every one of them rounded or cut by less than a unit of 2^-23
        assert rel(out[lo:hi], torch.stack(want)) < 5e-7 and rel(state[slots[i]], S) < 5e-7
    assert bool((out[n:] == 7.0).all()) and torch.equal(state[0], first[0])


@pytest.mark.parametrize("heads, dim, vdim", [(40, 16, 8), (16, 64, 64), (20, 48, 72), (8, 128, 200), (16, 96, 64)])
@pytest.mark.parametrize("lengths", [[65, 129, 640], [1000, 1, 64, 700]])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_memory_chunks(heads, dim, vdim, lengths, dtype):
    torch.manual_seed(dim + vdim)
    starts, slots, seq_start, slot_ids = step(lengths)
    n, wide = starts[-1], heads * (2 * dim + vdim)
    proj = torch.randn(n, wide + 2 * heads, device=DEV).to(dtype)
    bias_i, bias_f = torch.randn(heads, device=DEV) - 1.0, torch.rand(heads, device=DEV) * 4.0 + 1.0
    s, m = torch.randn(len(lengths) + 1, heads, dim, vdim, device=DEV), torch.zeros(len(lengths) + 1, heads, device=DEV)
    nn = torch.randn(len(lengths) + 1, heads, dim, device=DEV)
    before, out = (s.clone(), nn.clone(), m.clone()), torch.full((n + 2, heads * vdim), 7.0, device=DEV)
    scratch = torch.full((kernels.mlstm_chunked_scratch_floats(n, len(lengths), max(lengths), heads, dim, vdim),), float("nan"), device=DEV)
    kernels.mlstm_scan(proj, (0, heads * dim, 2 * heads * dim, wide, wide + heads), bias_i, bias_f, 15.0, dim ** -0.5, s, nn, m, slot_ids,
                       seq_start, out[:n], n_seqs=len(lengths), n_heads=heads, dim=dim, vdim=vdim, max_new=max(lengths), scratch=scratch)
    x = proj.to(F64)
    for i, (lo, hi) in enumerate(zip(starts[:-1], starts[1:])):
        q, k, v = (x[lo:hi, a:b].reshape(hi - lo, heads, -1) for a, b in
                   ((0, heads * dim), (heads * dim, 2 * heads * dim), (2 * heads * dim, wide)))
        a = 15.0 * torch.tanh((x[lo:hi, wide:wide + heads] + bias_i.to(F64)) / 15.0)
        b = torch.nn.functional.logsigmoid(15.0 * torch.tanh((x[lo:hi, wide + heads:] + bias_f.to(F64)) / 15.0))
        S, N, top = (t[slots[i]].to(F64) for t in before)
        want, size = [], []
        for t in range(hi - lo):
            new = torch.maximum(b[t] + top, a[t])
            keep, take = torch.exp(b[t] + top - new), torch.exp(a[t] - new)
            S = keep[:, None, None] * S + take[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
            N, top = keep[:, None] * N + take[:, None] * k[t], new
            qt = q[t] * dim ** -0.5
            div = torch.maximum((N * qt).sum(-1).abs(), torch.exp(-top)) + 1e-6
            want.append((torch.einsum("hkv,hk->hv", S, qt) / div[:, None]).reshape(-1))
            # what a 32-bit error of the divisor's sum, of |N| |q| units, makes of the result
            size.append((want[-1].reshape(heads, vdim) * (1.0 + N.norm(dim=-1) * qt.norm(dim=-1) / div)[:, None]).reshape(-1))
        err = out[lo:hi].to(F64) - torch.stack(want)
        assert float(err.norm() / torch.stack(size).norm()) < 2e-6
        assert rel(s[slots[i]], S) < 2e-6 and rel(nn[slots[i]], N) < 2e-6
    assert bool((out[n:] == 7.0).all()) and all(torch.equal(t[0], u[0]) for t, u in zip((s, nn, m), before))
