"""The short convolution over long runs: sequences that begin at, just before and just behind a block's first token, runs shorter
than the taps between longer ones, channels past a block, inputs kept from the step before."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("channels", [1, 255, 300])
@pytest.mark.parametrize("lengths", [[16, 16, 40], [15, 1, 2, 1, 30], [17, 3, 60], [65]])
@pytest.mark.parametrize("dtype, tol", [(torch.float32, 1e-6), (torch.bfloat16, 2.0 ** -8)])
def test_long_runs(taps, channels, lengths, dtype, tol):
    n = sum(lengths)
    src = torch.randn(n, channels, device=DEV).to(dtype)
    w, bias = torch.randn(channels, taps, device=DEV), torch.randn(channels, device=DEV)
    kept = torch.randn(len(lengths) + 2, taps - 1, channels, device=DEV)
    state = kept.clone()
    slots = torch.tensor([len(lengths) - i for i in range(len(lengths))], dtype=torch.int32, device=DEV)
    starts = torch.tensor([sum(lengths[:i]) for i in range(len(lengths) + 1)], dtype=torch.int32, device=DEV)
    token_seq = torch.cat([torch.full((m,), i) for i, m in enumerate(lengths)]).to(torch.int32).to(DEV)
    out = torch.empty(n, channels, device=DEV, dtype=dtype)
    kernels.short_conv(src, w, bias, state, slots, starts, token_seq, out, n_tokens=n, n_seqs=len(lengths), activation="swish")
    at = 0
    for i, m in enumerate(lengths):
        rows = torch.cat([kept[int(slots[i])].double(), src[at:at + m].double()])
        y = sum(rows[j:j + m] * w[:, j].double() for j in range(taps)) + bias.double()
        want = torch.nn.functional.silu(y)
        assert float((out[at:at + m].double() - want).norm() / want.norm()) < tol
        assert torch.equal(state[int(slots[i])], rows[m:].float())
        at += m
