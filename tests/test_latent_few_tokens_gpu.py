"""The steps before and after the latent attention of few tokens on tensor cores: tails of their blocks of 64 and 8 tokens, one block of 64
latent channels and several, rotated channels fewer than a head's, a layer with its own latent row and one without; splits of which one
saw no key.  Against 64 bits."""
import numpy as np
import plain_sovozen as plain
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


def dev(x):
    return torch.tensor(np.asarray(x), dtype=torch.float32, device=DEV).to(torch.bfloat16)


def host(x):
    return x.double().cpu().numpy()


def rel(got, want):
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


@pytest.mark.parametrize("dim, rank, rot, dims", [(16, 64, 16, 16), (64, 512, 64, 32), (48, 128, 6, 4)])
@pytest.mark.parametrize("n", [1, 63, 64, 65])
@pytest.mark.parametrize("owns", [False, True])
def test_before(dim, rank, rot, dims, n, owns):
    rng = np.random.default_rng(n + dim)
    heads, q_off = 3, 2
    lat_off = q_off + heads * (dim + rot) + 1
    proj = dev(rng.standard_normal((n, (lat_off + rank + rot + 1) // 2 * 2)))
    uk = dev(rng.standard_normal((heads, dim, rank)) / np.sqrt(dim))
    weight = torch.tensor(rng.uniform(0.5, 1.5, rank), dtype=torch.float32, device=DEV)
    freq = torch.tensor([30.0 ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float32, device=DEV)
    positions = rng.integers(0, 256, n).astype(np.int32)
    table = rng.permutation(4 * n + 1)[:4 * n].reshape(n, 4).astype(np.int32)      # (a sequence a token: no two file in one row)
    pool = torch.full((4 * n + 1, 64, rank + rot), 5.0, dtype=torch.bfloat16, device=DEV)
    q_latent = torch.zeros((n + 1, heads * (rank + rot)), dtype=torch.bfloat16, device=DEV)
    kernels.latent_decode_prep(proj, q_off, lat_off, uk, weight if owns else None, 1e-4, torch.tensor(positions, device=DEV),
                               torch.arange(n, dtype=torch.int32, device=DEV), freq, dims, torch.tensor(table, device=DEV), 4, pool,
                               q_latent, n_tokens=n, n_heads=heads, dim=dim, rank=rank, rot=rot, owns=owns)
    p, at = host(proj), positions % 64
    q = p[:, q_off:q_off + heads * (dim + rot)].reshape(n, heads, dim + rot)
    got = host(q_latent[:n]).reshape(n, heads, rank + rot)
    # bfloat16 results of 32-bit sums: half a unit of 2^-8 at most, a third of that in the norm
    assert rel(got[:, :, :rank], np.einsum("thd,hdr->thr", q[:, :, :dim], host(uk))) < 2.5e-3
    assert rel(got[:, :, rank:], plain.rotate_interleaved(q[:, :, dim:], positions, dims, 30.0)) < 2.5e-3
    assert bool((q_latent[n:] == 0).all())
    written = torch.zeros_like(pool, dtype=torch.bool)
    if owns:
        lat, page = p[:, lat_off:lat_off + rank + rot], table[np.arange(n), positions // 64]
        filed = host(pool[page, at])
        assert rel(filed[:, :rank], plain.rms_norm(lat[:, :rank], host(weight), 1e-4)) < 2.5e-3
        assert rel(filed[:, rank:], plain.rotate_interleaved(lat[:, rank:], positions, dims, 30.0)) < 2.5e-3
        written[page, at] = True
    assert bool((pool[~written] == 5.0).all())


def partial_results(rng, n, heads, splits, rank):
    sums, maxima = rng.standard_normal((n, heads, splits, rank)), rng.standard_normal((n, heads, splits)) * 3.0
    denoms = rng.uniform(0.5, 2.0, (n, heads, splits))
    maxima[:, :, 1], sums[:, :, 1], denoms[:, :, 1] = -np.inf, 0.0, 0.0      # a split that saw no key
    part = np.concatenate([sums, maxima[..., None], denoms[..., None]], axis=-1).astype(np.float32)
    sums, maxima, denoms = part[..., :rank].astype(np.float64), part[..., rank].astype(np.float64), part[..., rank + 1].astype(np.float64)
    w = np.where(np.isfinite(maxima), np.exp(maxima - maxima.max(axis=-1, keepdims=True)), 0.0)
    return torch.tensor(part.reshape(-1), device=DEV), (sums * w[..., None]).sum(axis=2) / (denoms * w).sum(axis=2)[..., None]


@pytest.mark.parametrize("rank, vdim", [(16, 16), (160, 48), (512, 64), (64, 32)])
@pytest.mark.parametrize("n", [1, 7, 8, 9])
@pytest.mark.parametrize("splits", [1, 5, 40])
@pytest.mark.parametrize("per_head", [False, True])
def test_after(rank, vdim, n, splits, per_head):
    rng = np.random.default_rng(rank + n + splits)
    heads = 3
    uv = dev(rng.standard_normal((heads, rank, vdim)) / np.sqrt(rank))
    gate = dev(rng.standard_normal((n, (heads if per_head else heads * vdim) + 6)))[:, 6:]
    out = torch.zeros((n + 1, heads * vdim), dtype=torch.bfloat16, device=DEV)
    if splits == 1:
        mixed = dev(rng.standard_normal((n, heads * rank)))
        merged = host(mixed).reshape(n, heads, rank)
        kernels.latent_decode_finish(uv, out, n_tokens=n, n_splits=1, mixed_latent=mixed, gate=gate)
    else:
        part, merged = partial_results(rng, n, heads, splits, rank)
        kernels.latent_decode_finish(uv, out, n_tokens=n, n_splits=splits, scratch=part, gate=gate)
    want = np.einsum("thr,hrv->thv", merged, host(uv)) * plain.sigmoid(host(gate).reshape(n, heads, -1))
    assert rel(host(out[:n]).reshape(n, heads, vdim), want) < 2.5e-3 and bool((out[n:] == 0).all())


def test_after_of_what_is_not_finite():
    """A latent channel that is infinite, or that bfloat16 would round to infinity: the results are those of multiply-adds."""
    rng = np.random.default_rng(3)
    n, heads, rank, vdim, splits = 9, 3, 64, 32, 4
    uv = dev(rng.uniform(0.5, 1.5, (heads, rank, vdim)) / rank)
    part, _ = partial_results(rng, n, heads, splits, rank)
    cells = part.view(n, heads, splits, rank + 2)
    cells[2, 1, 0, 7], cells[8, 0, 2, 63], cells[4, 2, 3, 20] = float("inf"), float("-inf"), float("nan")
    cells[5, 1, 0, 9], cells[5, 1, :, rank], cells[5, 1, 0, rank + 1] = 3.4e38, -30.0, 1.0
    cells[5, 1, 0, rank] = 0.0
    out = torch.empty((n, heads * vdim), dtype=torch.bfloat16, device=DEV)
    kernels.latent_decode_finish(uv, out, n_tokens=n, n_splits=splits, scratch=part)
    out = out.view(n, heads, vdim)
    assert bool((out[2, 1] == float("inf")).all()) and bool((out[8, 0] == float("-inf")).all()) and bool(torch.isnan(out[4, 2]).all())
    want = 3.4e38 * uv[1, 9].double()
    assert float(((out[5, 1].double() - want) / want).abs().max()) < 2.0 ** -8
    out[2, 1], out[8, 0], out[4, 2], out[5, 1] = 0.0, 0.0, 0.0, 0.0
    assert bool(torch.isfinite(out).all())
