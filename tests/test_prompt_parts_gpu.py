"""The 32-bit prompt attention on tensor cores in exact parts: the head sizes it takes, blocks of 64 queries and tiles of 64 keys at their
edges, windows, shared key heads, scattered pages and a step's own rows, against float64 and against the multiply-add kernel."""
import pytest
import torch
from test_prompt_queries_gpu import RUNS, attend

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
LONG = [(0, 64), (1, 63), (64, 65), (100, 129), (300, 1), (200, 8), (200, 9)]


def reference(q, k, v, past, window, causal=True):
    pos, j = past + torch.arange(q.shape[1], device=DEV)[:, None], torch.arange(k.shape[1], device=DEV)[None, :]
    seen = (j <= pos) if causal else torch.ones_like(j <= pos)
    seen = seen & (pos - j < window) if window else seen
    p = torch.softmax((q @ k.transpose(1, 2) * q.shape[2] ** -0.5).masked_fill(~seen, float("-inf")), -1)
    return (p @ v).transpose(0, 1).reshape(q.shape[1], -1)


@pytest.mark.parametrize("runs", [RUNS["one"], RUNS["edges"], LONG])
@pytest.mark.parametrize("hd", [16, 32, 48, 64])
@pytest.mark.parametrize("window", [0, 70])
def test_pages(runs, hd, window):
    out, proj, keys, values = attend(torch.float32, hd, runs, 1, window)
    at = 0
    for i, (past, new) in enumerate(runs):
        q = proj[at:at + new, :4 * hd].double().view(new, 4, hd).transpose(0, 1)
        k, v = (t[i, :past + new].double().transpose(0, 1).repeat_interleave(2, 0) for t in (keys, values))
        want = reference(q, k, v, past, window)
        # 32-bit sums of up to some hundred products and one exponential a key
        assert float((out[at:at + new].double() - want).norm() / want.norm()) < 1e-6
        at += new
    assert torch.equal(attend(torch.float32, hd, runs, 3, window)[0], out.repeat(3, 1))


@pytest.mark.parametrize("hd", [16, 48, 64])
@pytest.mark.parametrize("causal", [True, False])
def test_own_rows(hd, causal):
    torch.manual_seed(hd)
    news, heads = [1, 64, 65, 200, 128], 3
    proj = torch.randn(sum(news), 3 * heads * hd, device=DEV)
    proj[:, :heads * hd] *= 4.0
    starts = torch.tensor([sum(news[:i]) for i in range(len(news) + 1)], dtype=torch.int32, device=DEV)
    out = torch.full((sum(news) + 2, heads * hd), 7.0, device=DEV)
    kernels.attention_prefill_simt(proj, out, starts, torch.zeros(len(news), dtype=torch.int32, device=DEV), len(news), max(news), heads,
                                   heads, hd, hd ** -0.5, causal=causal, k_offset=heads * hd, v_offset=2 * heads * hd)
    at = 0
    for n in news:
        q, k, v = (proj[at:at + n, j * heads * hd:(j + 1) * heads * hd].double().view(n, heads, hd).transpose(0, 1) for j in range(3))
        want = reference(q, k, v, 0, 0, causal)
        assert float((out[at:at + n].double() - want).norm() / want.norm()) < 2e-6
        at += n
    assert bool((out[at:] == 7.0).all())


def test_what_is_no_number_comes_out_as_from_multiply_adds():
    torch.manual_seed(5)
    n, heads, hd = 150, 2, 64
    proj = torch.randn(n, 3 * heads * hd, device=DEV)
    proj[20, heads * hd + 3], proj[0, 2 * heads * hd + 20], proj[90, 5], proj[140, 70] = float("inf"), float("-inf"), float("nan"), 3.4e38
    starts, past = torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    shifted = torch.zeros(proj.numel() + 1, device=DEV)[1:].view_as(proj).copy_(proj)      # off the 16-byte boundaries
    out, want = torch.empty(n, heads * hd, device=DEV), torch.empty(n, heads * hd, device=DEV)
    for rows, into in ((proj, out), (shifted, want)):
        kernels.attention_prefill_simt(rows, into, starts, past, 1, n, heads, heads, hd, hd ** -0.5, k_offset=heads * hd, v_offset=2 * heads * hd)
    assert bool(torch.isfinite(want[:20, :20]).all()) and bool((want == float("-inf")).any()) and bool(torch.isnan(want[90, :hd]).all())
    torch.testing.assert_close(out, want, rtol=1e-5, atol=1e-5, equal_nan=True)
