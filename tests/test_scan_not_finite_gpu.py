"""Long runs of the selective scan, and its step sizes, at the ends of the numbers' range and beside large ones, against 64 bits."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda", torch.float64


def scan(dtype, inner, n_state, x, z, state):
    total = x.shape[0]
    gen = torch.Generator(device=DEV).manual_seed(n_state)
    low = torch.rand(total, 2 * n_state, generator=gen, device=DEV).add(0.5).to(dtype)
    dt, a_log, d_skip = torch.full((total, inner), 0.125, device=DEV), torch.zeros(inner, n_state, device=DEV), torch.ones(inner, device=DEV)
    out = torch.empty(total, inner, dtype=dtype, device=DEV)
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    _, _, need = kernels.selective_scan_pieces(total, total, 1, inner, n_state)
    kernels.selective_scan(x, z, dt, low, 0, n_state, a_log, d_skip, state, ints(0), ints(0, total), out, n_seqs=1, max_new=total,
                           scratch=torch.empty(need, device=DEV))
    S, want = torch.zeros(inner, n_state, device=DEV, dtype=F64), []
    for t in range(total):
        S = torch.exp(dt[t, :, None].to(F64) * -1.0) * S + (dt[t].to(F64) * x[t].to(F64))[:, None] * low[t, None, :n_state].to(F64)
        want.append(((S * low[t, None, n_state:].to(F64)).sum(-1) + x[t].to(F64)) * z[t].to(F64) / (1.0 + torch.exp(-z[t].to(F64))))
    return out.to(F64), torch.stack(want), S


@pytest.mark.parametrize("n_state", [1, 7, 8, 9, 15, 16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_an_infinite_row(n_state, dtype):
    inner, total = 70, 200
    x, z = torch.ones(total, inner, device=DEV, dtype=dtype), torch.ones(total, inner, device=DEV, dtype=dtype)
    x[90, 3], x[150, 69] = float("inf"), float("-inf")
    state = torch.zeros(1, inner, n_state, device=DEV)
    out, want, S = scan(dtype, inner, n_state, x, z, state)
    ok = torch.isfinite(want)
    assert torch.equal(out[~ok], want[~ok]) and float(((out - want).abs()[ok] / want[ok]).max()) < 2.0 ** -8
    ok = torch.isfinite(S)
    assert torch.equal(state[0].to(F64)[~ok], S[~ok]) and float(((state[0].to(F64) - S).abs()[ok] / S[ok]).max()) < 1e-5


@pytest.mark.parametrize("n_state", [7, 8, 16])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_gate_far_below_zero(n_state, dtype):
    inner, total = 70, 200
    z = torch.tensor([-1.0, -20.0, -60.0, -85.0, -87.5, -88.0, -88.5], device=DEV).to(dtype).repeat(total * inner // 7).view(total, inner)
    x = torch.full((total, inner), 1e30, device=DEV, dtype=dtype)
    out, want, _ = scan(dtype, inner, n_state, x, z, torch.zeros(1, inner, n_state, device=DEV))
    # (the gates themselves are down to 2^-120, with all of their bits)
    assert float(((out - want).abs() / want.abs()).max()) < (2.0 ** -8 if dtype is torch.bfloat16 else 1e-5)


@pytest.mark.parametrize("rank", [32, 48, 64])
def test_step_sizes_beside_a_large_channel(rank):
    torch.manual_seed(rank)
    low, w = torch.rand(640, rank, device=DEV) + 0.5, torch.rand(512, rank, device=DEV) + 0.5
    low[:, 0] = 4096.0
    low, dt = low.bfloat16(), torch.empty(640, 512, device=DEV)
    kernels.selective_scan_dt(low, w, torch.zeros(512, device=DEV), dt, n_tokens=640)
    want = low.to(F64) @ w.to(F64).T      # (a softplus of thousands is its argument)
    # the sum of the large channel's 16 is cut once, by 2^-23 at most, and the up to three others are added with a rounding each
    assert float(((dt.to(F64) - want) / want).pow(2).mean().sqrt()) < 2.0 ** -22.5
