"""The 32-bit product and prompt attention at the edges of their tiles, against float64."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"
# 32-bit sums of up to 1,000 products, each rounded once: well under sqrt(1000) half units in the last place
TOL = 2e-6


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("m", [1, 15, 16, 17, 32, 33, 63, 64, 65, 200, 801])
@pytest.mark.parametrize("n, k", [(4, 4), (32, 32), (36, 28), (100, 36), (768, 1000)])
@pytest.mark.parametrize("nk", [False, True])
def test_product_at_the_edges_of_its_tiles(m, n, k, nk):
    a, w = torch.randn(m, k, device=DEV), torch.randn(k, n, device=DEV)
    bias, res = torch.randn(n, device=DEV), torch.randn(m, n, device=DEV)
    w_arg = w.t().contiguous() if nk else w
    out = torch.full((m + 2, n), 7.0, device=DEV)
    kernels.linear_simt(a, w_arg, bias, out, m=m, w_is_nk=nk, activation="gelu_new", residual=torch.cat([res, res[:1], res[:1]]))
    want = torch.nn.functional.gelu(a.double() @ w.double() + bias.double(), approximate="tanh") + res.double()
    assert rel(out[:m], want) < TOL
    assert float((out[m:] - 7.0).abs().max()) == 0.0


def test_product_of_a_row_does_not_depend_on_the_other_rows():
    a, w = torch.randn(801, 768, device=DEV), torch.randn(768, 96, device=DEV)
    whole, alone = torch.empty(801, 96, device=DEV), torch.empty(1, 96, device=DEV)
    kernels.linear_simt(a, w, None, whole)
    kernels.linear_simt(a[800:].contiguous(), w, None, alone)
    assert torch.equal(whole[800:], alone)


@pytest.mark.parametrize("shift", [1, 2, 4])
@pytest.mark.parametrize("nk", [False, True])
def test_product_of_operands_off_a_16_byte_boundary(shift, nk):
    def off(x):
        flat = torch.empty(x.numel() + shift, device=DEV)
        flat[shift:] = x.reshape(-1)
        return flat[shift:].view(x.shape)

    a, w, bias, res = (torch.randn(s, device=DEV) for s in ((33, 64), (64, 64), (64,), (33, 64)))
    want = a.double() @ w.double() + bias.double() + res.double()
    w_arg = w.t().contiguous() if nk else w
    for operands in ((off(a), w_arg, bias, res), (a, off(w_arg), bias, res), (a, w_arg, off(bias), res), (a, w_arg, bias, off(res))):
        out = off(torch.empty(33, 64, device=DEV))
        kernels.linear_simt(operands[0], operands[1], operands[2], out, w_is_nk=nk, residual=operands[3])
        assert rel(out, want) < TOL


@pytest.mark.parametrize("hd", [3, 6, 64, 68, 100, 200, 256])
@pytest.mark.parametrize("window", [0, 1, 40])
def test_attention_at_the_edges_of_its_tiles(hd, window):
    news, heads, kv_heads = [1, 31, 32, 33, 64, 65, 130], 4, 2
    width = (heads + 2 * kv_heads) * hd
    proj = torch.randn(sum(news), width, device=DEV)
    starts = torch.tensor([sum(news[:i]) for i in range(len(news) + 1)], dtype=torch.int32, device=DEV)
    out = torch.empty(sum(news), heads * hd, device=DEV)
    kernels.attention_prefill_simt(proj, out, starts, torch.zeros(len(news), dtype=torch.int32, device=DEV), len(news), max(news),
                                   heads, kv_heads, hd, hd ** -0.5, window=window, k_offset=heads * hd,
                                   v_offset=(heads + kv_heads) * hd)
    at = 0
    for n in news:
        rows = proj[at:at + n].double()
        q = rows[:, :heads * hd].view(n, heads, hd).transpose(0, 1)
        k = rows[:, heads * hd:(heads + kv_heads) * hd].view(n, kv_heads, hd).transpose(0, 1).repeat_interleave(2, 0)
        v = rows[:, (heads + kv_heads) * hd:].view(n, kv_heads, hd).transpose(0, 1).repeat_interleave(2, 0)
        i, j = torch.arange(n, device=DEV)[:, None], torch.arange(n, device=DEV)[None, :]
        seen = (j <= i) & ((i - j < window) if window else True)
        p = torch.softmax((q @ k.transpose(1, 2) * hd ** -0.5).masked_fill(~seen, float("-inf")), -1)
        assert rel(out[at:at + n], (p @ v).transpose(0, 1).reshape(n, -1)) < TOL
        at += n
