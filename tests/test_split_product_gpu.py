"""The 32-bit product on tensor cores in exact parts: the edges of its tiles of 128 x 64 and of its k-blocks of 64, every number of
blocks a tile, against float64 and against itself; numbers that are not finite, and those that a part would round to one."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(got, want):
    return float((got.double() - want).norm() / want.norm())


@pytest.mark.parametrize("m", [1, 127, 128, 129, 300])
@pytest.mark.parametrize("n, k", [(256, 768), (260, 772), (300, 1000), (768, 3072), (2048, 2048)])
@pytest.mark.parametrize("nk", [False, True])
def test_product_in_parts(m, n, k, nk):
    torch.manual_seed(m + n)
    a, w = torch.randn(m, k, device=DEV), torch.randn(k, n, device=DEV) * k ** -0.5
    bias, res = torch.randn(n, device=DEV), torch.randn(m, n, device=DEV)
    w_arg = w.t().contiguous() if nk else w
    product = a.double() @ w.double()
    seen = []
    for split in (0, 1, 2, 4, 8):
        out = torch.full((m + 2, n), 7.0, device=DEV)
        kernels.linear_simt(a, w_arg, None, out, m=m, w_is_nk=nk, split=split)
        # some dozen additions of 32-bit sums, each rounded once or cut: less than the multiply-adds' chain of hundreds
        assert rel(out[:m], product) < 2e-7 and bool((out[m:] == 7.0).all())
        seen.append(out)
    assert all(torch.equal(seen[0], other) for other in seen[1:])
    want, seen_res = torch.nn.functional.gelu(product + bias.double(), approximate="tanh") + res.double(), []
    for split in (0, 1, 2, 4, 8):
        out = torch.full((m + 2, n), 7.0, device=DEV)
        out[:m] = res
        kernels.linear_simt(a, w_arg, bias, out, m=m, w_is_nk=nk, activation="gelu_new", residual=out, split=split)      # in place
        assert rel(out[:m], want) < 5e-7 and bool((out[m:] == 7.0).all())
        seen_res.append(out)
    assert all(torch.equal(seen_res[0], other) for other in seen_res[1:])
    alone = torch.empty(1, n, device=DEV)
    kernels.linear_simt(a[m - 1:].contiguous(), w_arg, None, alone, w_is_nk=nk)
    assert torch.equal(alone[0], seen[0][m - 1])
    kernels.check_status(a.device)


@pytest.mark.parametrize("split", [1, 4])
def test_epilogue(split):
    torch.manual_seed(1)
    a, w, bias, res = torch.randn(130, 768, device=DEV), torch.randn(768, 260, device=DEV), torch.randn(260, device=DEV), torch.randn(130, 260, device=DEV)
    want = torch.nn.functional.gelu(a.double() @ w.double() + bias.double(), approximate="tanh") + res.double()
    kernels.linear_simt(a, w, bias, res, activation="gelu_new", residual=res, split=split)      # in place
    assert rel(res, want) < 5e-7


@pytest.mark.parametrize("split", [1, 2, 8])
def test_what_is_not_finite(split):
    torch.manual_seed(2)
    a, w = torch.randn(200, 768, device=DEV), torch.randn(768, 256, device=DEV).abs() + 0.1
    a[3, 10], a[50, 700], a[60, 5], a[61, 6] = float("inf"), float("-inf"), float("nan"), 3.4e38
    a[70] = 1e-42
    out = torch.empty(200, 256, device=DEV)
    kernels.linear_simt(a, w, None, out, split=split)
    assert bool((out[3] == float("inf")).all()) and bool((out[50] == float("-inf")).all()) and bool(torch.isnan(out[60]).all())
    want = (a.double() @ w.double()).float()
    same = torch.isfinite(want) & torch.isfinite(out)
    assert torch.equal(torch.isfinite(want[61]), torch.isfinite(out[61])) and bool(((out[61] - want[61]).abs() <= 1e-5 * want[61].abs())[same[61]].all())
    assert float((out[70] - want[70]).abs().max()) < 1e-38
    rest = [r for r in range(200) if r not in (3, 50, 60, 61, 70)]
    assert rel(out[rest], a[rest].double() @ w.double()) < 2e-7


def test_a_profile_shows_the_product_alone():
    a, w, out = torch.randn(5, 1076, device=DEV), torch.randn(1076, 1052, device=DEV), torch.empty(5, 1052, device=DEV)
    with kernels.KernelProfile() as profile:      # (a size that no other test has asked for: the first question is asked here)
        kernels.linear_simt(a, w, None, out)
    (row,) = profile.summary()
    assert row["kernel"] == "linear_split" and row["flops"] == 2.0 * 5 * 1052 * 1076


@pytest.mark.parametrize("split", [0, 1, 8])
def test_rows_of_no_whole_pieces(split):
    torch.manual_seed(3)
    a, w = torch.randn(130, 772, device=DEV), torch.randn(257, 772, device=DEV) * 772 ** -0.5      # ([N,K]: N is free)
    bias, out = torch.randn(257, device=DEV), torch.full((132, 257), 7.0, device=DEV)
    kernels.linear_simt(a, w, bias, out, m=130, w_is_nk=True, split=split)
    assert rel(out[:130], a.double() @ w.double().T + bias.double()) < 2e-7 and bool((out[130:] == 7.0).all())
