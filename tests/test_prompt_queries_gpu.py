"""The 32-bit prompt attention with 8, 16 and 32 queries a block, against float64 and against one another: one token behind many,
runs at the blocks' edges, keys at the tiles' edges, pages that lie scattered, windows, heads off 16-byte boundaries."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
# the sequences' (tokens before, tokens of the step); how often they are repeated decides how many queries a block takes
RUNS = {"one": [(0, 1), (63, 1), (64, 1), (200, 1)], "few": [(0, 7), (60, 8), (130, 5)], "edges": [(0, 9), (50, 16), (127, 13)],
        "long": [(0, 17), (3, 33), (129, 40), (0, 65)]}


def attend(dtype, hd, runs, copies, window):
    heads, kv_heads = 4, 2
    runs = runs * copies
    pasts, news = [r[0] for r in runs], [r[1] for r in runs]
    n, per = sum(news), max(-(-(p + m) // 64) for p, m in runs)
    gen = torch.Generator(device=DEV).manual_seed(7)
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV).to(dtype)  # noqa: E731
    one = len(runs) // copies
    first = rand(sum(news[:one]), (heads + 2 * kv_heads) * hd)
    proj = first.repeat(copies, 1).contiguous()
    keys, values = rand(one, per * 64, kv_heads, hd), rand(one, per * 64, kv_heads, hd)
    table = torch.randperm(len(runs) * per, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(len(runs), per).to(DEV)
    k_pool, v_pool = torch.zeros(2, len(runs) * per, kv_heads, 64, hd, dtype=dtype, device=DEV).unbind(0)
    for pool, rows in ((k_pool, keys), (v_pool, values)):
        pool[table.long().view(-1)] = rows.repeat(copies, 1, 1, 1).view(len(runs) * per, 64, kv_heads, hd).transpose(1, 2)
    starts = torch.tensor([sum(news[:i]) for i in range(len(news) + 1)], dtype=torch.int32, device=DEV)
    out = torch.empty(n, heads * hd, dtype=dtype, device=DEV)
    kernels.attention_prefill_simt(proj, out, starts, torch.tensor(pasts, dtype=torch.int32, device=DEV), len(runs), max(news), heads,
                                   kv_heads, hd, hd ** -0.5, window=window, k_pool=k_pool, v_pool=v_pool, table=table, table_len=per)
    return out, proj, keys, values


@pytest.mark.parametrize("runs", list(RUNS))
@pytest.mark.parametrize("hd", [3, 20, 64, 80, 192, 256])
@pytest.mark.parametrize("window", [0, 50])
@pytest.mark.parametrize("dtype, tol", [(torch.float32, 2e-6), (torch.bfloat16, 2.0 ** -8)])      # (32-bit sums; one rounding to 8 bits)
def test_queries_a_block(runs, hd, window, dtype, tol):
    few = attend(dtype, hd, RUNS[runs], 1, window)
    out, proj, keys, values = few
    at = 0
    for i, (past, new) in enumerate(RUNS[runs]):
        q = proj[at:at + new, :4 * hd].double().view(new, 4, hd).transpose(0, 1)
        k, v = (t[i, :past + new].double().transpose(0, 1).repeat_interleave(2, 0) for t in (keys, values))
        pos, j = past + torch.arange(new, device=DEV)[:, None], torch.arange(past + new, device=DEV)[None, :]
        seen = (j <= pos) & ((pos - j < window) if window else True)
        p = torch.softmax((q @ k.transpose(1, 2) * hd ** -0.5).masked_fill(~seen, float("-inf")), -1)
        want = (p @ v).transpose(0, 1).reshape(new, -1)
        assert float((out[at:at + new].double() - want).norm() / want.norm()) < tol
        at += new
    for copies in (20, 60):      # more sequences, more queries a block: the same numbers
        many = attend(dtype, hd, RUNS[runs], copies, window)[0]
        assert torch.equal(many, out.repeat(copies, 1))
