"""The prompt attention that files the step's own keys and values in the pages: whole pages, pages that a sequence leaves unfilled, shared
key heads, windows, both head sizes; beside kv_append and the attention without it, bit for bit, and nothing else written."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("heads,kv_heads", [(4, 4), (6, 2)])
@pytest.mark.parametrize("news", [[1], [64], [63, 65, 128, 1], [127, 129, 300, 191, 192, 64]])
@pytest.mark.parametrize("window", [0, 100])
def test_files_what_the_append_writes(hd, heads, kv_heads, news, window):
    torch.manual_seed(7)
    n, seqs, per = sum(news), len(news), max(-(-m // 64) for m in news) + 1
    q_width, kv_width = heads * hd, kv_heads * hd
    proj = torch.randn(n, q_width + 2 * kv_width, device=DEV).bfloat16()
    ints = dict(dtype=torch.int32, device=DEV)
    starts = torch.tensor([sum(news[:i]) for i in range(seqs + 1)], **ints)
    zero, lens = torch.zeros(seqs, **ints), torch.tensor(news, **ints)
    positions = torch.cat([torch.arange(m, **ints) for m in news])
    token_seq = torch.cat([torch.full((m,), i, **ints) for i, m in enumerate(news)])
    table = torch.randperm(seqs * per + 2, device=DEV)[:seqs * per].to(torch.int32).view(seqs, per)
    pools = [[torch.full((seqs * per + 2, kv_heads, 64, hd), 7.0, device=DEV, dtype=torch.bfloat16) for _ in range(2)] for _ in range(2)]
    outs = [torch.empty(n, q_width, device=DEV, dtype=torch.bfloat16) for _ in range(2)]
    args = (starts, zero, seqs, max(news), heads, kv_heads, hd, hd ** -0.5)
    where = dict(window=window, k_offset=q_width, v_offset=q_width + kv_width)
    assert kernels.attention_prefill_files(proj, pools[0][0], hd, True)
    kernels.kv_append(proj, q_width, q_width + kv_width, positions, token_seq, lens, table, per, *pools[0], n, kv_heads, hd)
    kernels.attention_prefill(proj, outs[0], *args, **where)
    kernels.attention_prefill(proj, outs[1], *args, file=(*pools[1], table), **where)
    assert all(torch.equal(a, b) for a, b in zip(pools[0], pools[1])) and torch.equal(*outs)
