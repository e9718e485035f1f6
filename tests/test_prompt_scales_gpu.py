"""The tcgen05 prompt attention at scales below zero and of zero, and over rows whose maximum grows from tile to tile by less than
what makes the earlier tiles vanish, in every pair of key and value sizes, against float64."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


def attend(q, k, v, scale, window):
    """q, k [n, heads, dq], v [n, heads, dv], one sequence."""
    n, heads, dv = v.shape
    out = torch.empty(n, heads, dv, dtype=torch.bfloat16, device=DEV)
    laid = [x.transpose(0, 1).contiguous().transpose(0, 1) for x in (k, v)]
    kernels.sink_attention(q, *laid, out, torch.tensor([0, n], dtype=torch.int32, device=DEV), n_seqs=1, max_new=n, scale=scale,
                           window=window, past_len=torch.zeros(1, dtype=torch.int32, device=DEV), impl="tcgen05")
    kernels.check_status(out.device)
    i, j = torch.arange(n, device=DEV)[:, None], torch.arange(n, device=DEV)[None, :]
    seen = (j <= i) & ((i - j < window) if window else True)
    s = torch.einsum("ihd,jhd->hij", q.double(), k.double()) * scale
    p = torch.softmax(s.masked_fill(~seen, float("-inf")), 2)
    return out.double(), torch.einsum("hij,jhd->ihd", p, v.double())


@pytest.mark.parametrize("dq", [64, 128])
@pytest.mark.parametrize("dv", [64, 128])
@pytest.mark.parametrize("window", [0, 200])
@pytest.mark.parametrize("scale", [-0.2, 0.0, 0.2])
def test_scales(dq, dv, window, scale):
    gen = torch.Generator(device=DEV).manual_seed(9)
    q, k, v = (torch.randn(700, 3, d, generator=gen, device=DEV).bfloat16() for d in (dq, dq, dv))
    got, want = attend(q, k, v, scale, window)
    assert float((got - want).norm() / want.norm()) < 2.0 ** -7      # (weights and results are rounded to 8 bits once each)


@pytest.mark.parametrize("dq", [64, 128])
@pytest.mark.parametrize("dv", [64, 128])
@pytest.mark.parametrize("growth", [3, 7, 9, 14])      # powers of two from tile to tile: the reference moves past 8
def test_rows_whose_maximum_grows(dq, dv, growth):
    n = 640
    gen = torch.Generator(device=DEV).manual_seed(10)
    noise = lambda d: torch.randn(n, 3, d, generator=gen, device=DEV)  # noqa: E731
    tile = (torch.arange(n, device=DEV) // 128).float()[:, None]
    q, k, v = 0.2 * noise(dq), 0.2 * noise(dq), noise(dv)
    q[:, :, 0], k[:, :, 0] = 1.0, growth * tile      # (a key's score in powers of two, exact in 8 bits)
    v = v * torch.exp2(-growth * tile)[:, :, None]      # (the tiles' shares of a row are of one size)
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    got, want = attend(q, k, v, 0.6931471805599453, 0)
    size = want.abs().amax((1, 2), keepdim=True)          # (rows of later tiles are smaller by what v shrinks: each row by its own size)
    assert float(((got - want) / size).norm() / (want / size).norm()) < 2.0 ** -6      # (shares of one size, each rounded to 8 bits, of either sign)
