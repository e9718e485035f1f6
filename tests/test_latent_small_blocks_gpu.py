"""The latent attention in blocks of 16 rows (one token a sequence, more blocks than multiprocessors), against float64 and against
the same sequences a few at a time, which take blocks of 64 rows; and how many runs a step's keys are cut into."""
import types

import pytest
import torch

from burn_transformers_b200 import kernels
from burn_transformers_b200.parts.latent_attention import LatentAttention

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rank, rot", [(24, 0), (64, 16), (128, 32), (256, 32), (512, 64)])
@pytest.mark.parametrize("heads", [1, 5, 16])
@pytest.mark.parametrize("seqs, runs", [(160, 1), (64, 4), (300, 3)])
@pytest.mark.parametrize("window, with_sink", [(0, True), (40, False)])
def test_one_token_a_sequence_in_small_blocks(rank, rot, heads, seqs, runs, window, with_sink):
    gen = torch.Generator(device=DEV).manual_seed(rank + heads)
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV)  # noqa: E731
    dk, scale = rank + rot, 0.7 * (rank + rot) ** -0.5
    past = torch.tensor([(0, 31, 32, 64, 200, 77)[i % 6] for i in range(seqs)], dtype=torch.int32, device=DEV)
    per = 4
    q, pool = rand(seqs, heads * dk).bfloat16(), rand(seqs * per, 64, dk).bfloat16()
    table = torch.randperm(seqs * per, generator=torch.Generator().manual_seed(2)).to(torch.int32).view(seqs, per).to(DEV)
    sink = rand(heads) if with_sink else None

    def attend(some):
        n = len(some)
        out = torch.empty(n, heads * rank, dtype=torch.bfloat16, device=DEV)
        scratch = torch.empty(max(1, kernels.latent_attention_scratch_floats(n, heads, rank, runs)), device=DEV)
        kernels.latent_attention(q[some].contiguous(), out, pool, table[some].contiguous(), per,
                                 torch.arange(n + 1, dtype=torch.int32, device=DEV), past[some].contiguous(), n_tokens=n, n_seqs=n,
                                 max_new=1, n_heads=heads, rank=rank, rot=rot, scale=scale, sink=sink, n_splits=runs,
                                 scratch=scratch, window=window)
        return out

    got = attend(torch.arange(seqs, device=DEV))
    few = torch.cat([attend(torch.arange(i, min(i + 10, 60), device=DEV)) for i in range(0, 60, 10)])
    rows = pool[table.long()].view(seqs, per * 64, dk).double()
    j, pos = torch.arange(per * 64, device=DEV)[None, :], past[:, None].long()
    seen = (j <= pos) & ((pos - j < window) if window else True)
    s = torch.einsum("bhd,bjd->bhj", q.double().view(seqs, heads, dk), rows) * scale
    s = s.masked_fill(~seen[:, None, :], float("-inf"))
    if with_sink:
        s = torch.cat([s, sink.double()[None, :, None].expand(seqs, heads, 1)], 2)
    p = torch.softmax(s, 2)[:, :, :per * 64]
    want = torch.einsum("bhj,bjr->bhr", p, rows[:, :, :rank]).reshape(seqs, -1)
    # (weights and results are rounded to 8 bits once each)
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -7
    assert float((few.double() - want[:60]).norm() / want[:60].norm()) < 2.0 ** -7
    # the same keys in the same order on the same instructions: the size of the block does not show
    assert torch.equal(got[:60], few)


def test_runs_of_keys_never_leave_the_two_numbers_around_two_blocks():
    part = LatentAttention(64, 16, 16, 8, 16, 512, 0.1, 1e-5, types.SimpleNamespace(rotates=True, dims=8))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for seqs in (1, 8, 50, 64, 100, sms, sms + 12, 2 * sms - 1, 2 * sms, 600):
        for bound in (33, 200, 1000):
            for dtype in (torch.float32, torch.bfloat16):
                ctx = types.SimpleNamespace(max_new=1, n_seqs=seqs, n_tokens=seqs, ctx_bound=bound, dtype=dtype,
                                            ws=types.SimpleNamespace(device=torch.device("cuda", 0)))
                runs = part._splits(ctx, 64)
                more, fewer = (max(1, min(n, -(-bound // 32), 64)) for n in (-(-2 * sms // seqs), 2 * sms // seqs))
                assert runs in (more, fewer) and (dtype == torch.bfloat16 or runs == more)
