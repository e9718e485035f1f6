"""Long runs of the selective scan with up to 16 state indices (a thread a channel), and the step sizes' kernel, at the edges of their
blocks: channels around 64 and 256, states that fill a thread's numbers or leave some idle, pieces of 64 tokens and of more, last
pieces of one token.  Against the recurrence in 64 bits."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("inner, n_state", [(64, 16), (65, 16), (63, 1), (130, 7), (64, 8), (1, 9), (200, 15)])
@pytest.mark.parametrize("lengths", [[65], [129, 1, 64, 70], [4200, 97]])
@pytest.mark.parametrize("dtype, tol", [(torch.float32, 1e-5), (torch.bfloat16, 2.0 ** -8)])
def test_pieces_equal_the_recurrence(inner, n_state, lengths, dtype, tol):
    gen = torch.Generator(device=DEV).manual_seed(inner * 31 + n_state)
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV)  # noqa: E731
    total, n_seqs = sum(lengths), len(lengths)
    starts = [sum(lengths[:i]) for i in range(n_seqs + 1)]
    seq_start = torch.tensor(starts, dtype=torch.int32, device=DEV)
    slots = torch.tensor([n_seqs - i for i in range(n_seqs)], dtype=torch.int32, device=DEV)
    xz, low = rand(total, 2 * inner + 3).to(dtype), rand(total, 2 * n_state + 5).to(dtype)
    x, z = xz[:, 1:1 + inner], xz[:, 2 + inner:2 + 2 * inner]
    dt = torch.nn.functional.softplus(rand(total, inner) - 3.0)
    a_log, d_skip, state = rand(inner, n_state) * 0.5 - 1.0, rand(inner), 3.0 * rand(n_seqs + 1, inner, n_state)
    out = torch.full((total + 2, inner), 7.0, dtype=dtype, device=DEV)
    S = [state[int(slots[i])].double() for i in range(n_seqs)]
    untouched = state[0].clone()
    piece, _, need = kernels.selective_scan_pieces(max(lengths), total, n_seqs, inner, n_state)
    assert piece > 0
    kernels.selective_scan(x, z, dt, low, 2, 3 + n_state, a_log, d_skip, state, slots, seq_start, out[:total], n_seqs=n_seqs,
                           out_scale=1.25, max_new=max(lengths), scratch=torch.full((need,), float("nan"), device=DEV))
    A, B, C = -torch.exp(a_log.double()), low[:, 2:2 + n_state].double(), low[:, 3 + n_state:3 + 2 * n_state].double()
    xd, zd, dd = x.double(), z.double(), dt.double()
    decay, feed = torch.exp(dd[:, :, None] * A), (dd * xd)[:, :, None] * B[:, None, :]
    want = torch.empty((total, inner), dtype=torch.float64, device=DEV)
    for i, (lo, hi) in enumerate(zip(starts[:-1], starts[1:])):
        for t in range(lo, hi):
            S[i] = decay[t] * S[i] + feed[t]
            want[t] = S[i] @ C[t]
        # (the state stays in 32 bits with either type: its error is that of some hundred roundings, decays of 2 units included)
        assert float((state[int(slots[i])].double() - S[i]).norm() / S[i].norm()) < 1e-5
    want = (want + d_skip.double() * xd) * zd * torch.sigmoid(zd) * 1.25
    assert float((out[:total].double() - want).norm() / want.norm()) < tol
    assert bool((out[total:] == 7.0).all()) and torch.equal(state[0], untouched)


@pytest.mark.parametrize("channels, rank", [(256, 16), (257, 4), (255, 3), (512, 48), (31, 160), (2, 1), (300, 129), (33, 18), (64, 64),
                                            (1024, 32), (96, 66), (1, 2)])
@pytest.mark.parametrize("n_tokens", [1, 15, 17, 2500])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_step_sizes(channels, rank, n_tokens, dtype):
    gen = torch.Generator(device=DEV).manual_seed(channels + rank)
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV)  # noqa: E731
    low, w, b = rand(n_tokens, rank + 3).to(dtype), rand(channels, rank) * rank ** -0.5, 4.0 * rand(channels)
    dt = torch.full((n_tokens + 2, channels), 7.0, device=DEV)
    kernels.selective_scan_dt(low, w, b, dt, n_tokens=n_tokens)
    want = torch.nn.functional.softplus(low[:, :rank].double() @ w.double().T + b.double(), threshold=200.0)
    # a 32-bit chain of `rank` multiply-adds on numbers of about one and a bias of four, then the softplus: relative to its size
    assert float((dt[:n_tokens].double() - want).abs().max()) < 1e-6 * (rank ** 0.5 + 16)
    assert float((dt[:n_tokens].double() - want).norm() / want.norm()) < 1e-6
    assert bool((dt[n_tokens:] == 7.0).all())


def test_step_sizes_of_an_infinite_row_are_infinite_or_zero():
    low, w, b = torch.zeros(20, 16, device=DEV).bfloat16(), torch.ones(64, 16, device=DEV), torch.zeros(64, device=DEV)
    w[1::2] = -1.0
    low[3, 5] = float("inf")
    dt = torch.empty(20, 64, device=DEV)
    kernels.selective_scan_dt(low, w, b, dt, n_tokens=20)
    assert bool((dt[3, 0::2] == float("inf")).all()) and bool((dt[3, 1::2] == 0.0).all())
    assert bool(torch.isfinite(dt[:3]).all()) and bool(torch.isfinite(dt[4:]).all())
