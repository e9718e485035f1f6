"""The selective scan's stored state while a run's pieces go side by side: every piece starts from a copy of it, since the last
piece, which may be a single token and the first to end, replaces it."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lengths", [[65], [129, 65, 7, 64, 193]])
@pytest.mark.parametrize("inner, n_state", [(2048, 16), (33, 70)])
@pytest.mark.parametrize("dtype, tol", [(torch.float32, 2e-5), (torch.bfloat16, 2.0 ** -8)])
def test_pieces_start_from_a_copy_of_the_state(lengths, inner, n_state, dtype, tol):
    gen = torch.Generator(device=DEV).manual_seed(5)
    rand = lambda *s: torch.randn(s, generator=gen, device=DEV)  # noqa: E731
    total, n_seqs = sum(lengths), len(lengths)
    starts = [sum(lengths[:i]) for i in range(n_seqs + 1)]
    seq_start = torch.tensor(starts, dtype=torch.int32, device=DEV)
    slots = torch.tensor([n_seqs - i for i in range(n_seqs)], dtype=torch.int32, device=DEV)
    x, z, low = rand(total, inner).to(dtype), rand(total, inner).to(dtype), rand(total, 2 * n_state).to(dtype)
    dt = torch.nn.functional.softplus(rand(total, inner) - 3.0)
    a_log, d_skip, first = rand(inner, n_state) * 0.5 - 1.0, rand(inner), 10.0 * rand(n_seqs + 1, inner, n_state)
    piece, _, need = kernels.selective_scan_pieces(max(lengths), total, n_seqs, inner, n_state)
    seen = []
    for cut in (False, True, True, True):
        state, out = first.clone(), torch.empty_like(x)
        scratch = torch.full((need,), float("nan"), device=DEV)
        kernels.selective_scan(x, z, dt, low, 0, n_state, a_log, d_skip, state, slots, seq_start, out, n_seqs=n_seqs,
                               **(dict(max_new=max(lengths), scratch=scratch) if cut else {}))
        seen.append((out, state, scratch))
    for i, n in enumerate(lengths):          # what the pieces read lies apart from what the last one writes
        count = -(-n // piece)
        cell = seen[1][2].view(-1, inner, n_state + 1)[starts[i] // piece + i + count - 1]
        if count > 1:
            assert torch.equal(cell[:, :n_state], first[int(slots[i])])
    for got in (0, 1):
        assert torch.equal(seen[1][got], seen[2][got]) and torch.equal(seen[1][got], seen[3][got])
        # (the joined pieces form the same sums in another order: a few roundings of the state, and one to the rows' type)
        assert float((seen[1][got].double() - seen[0][got].double()).norm() / seen[0][got].double().norm()) < tol
