"""The gated product (a gate's and an up matrix's rows in one tcgen05 product, the pair formed on the way out) at the edges of its
tiles: rows around 128 and 256, results that are no whole chunks of 32 or pieces of 8 columns, against float64."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV = "cuda"


def paired(g, u, rule, limit):
    if rule == "swish_clamp":
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        return g * torch.sigmoid(1.702 * g) * (u + 1.0)
    if rule == "swish":
        return g * torch.sigmoid(g) * u
    return torch.nn.functional.gelu(g, approximate="tanh" if rule == "gelu_new" else "none") * u


@pytest.mark.parametrize("m", [1, 65, 127, 128, 129, 256, 257, 1030, 5000])
@pytest.mark.parametrize("inner, k", [(8, 8), (30, 64), (32, 72), (100, 200), (160, 1024), (2816, 136)])
def test_gated_product(m, inner, k):
    torch.manual_seed(m + inner)
    a = torch.randn(m, k, device=DEV).bfloat16()
    w = (torch.randn(2 * inner, k, device=DEV) * 2.0 * k ** -0.5).bfloat16()
    both = a.double() @ w.double().T
    for rule, limit in (("gelu_new", 0.0), ("gelu", 0.0), ("swish", 0.0), ("swish_clamp", 1.5)):
        out = torch.full((m + 2, inner), 3.0, device=DEV).bfloat16()
        kernels.gated_tcgen05(a, w, out, m=m, activation=rule, limit=limit)
        want = paired(both[:, :inner], both[:, inner:], rule, limit)
        # one rounding to bfloat16 of each result: half a unit of 2^-7, so 2^-8 of its size at most, and less than 2^-9 in the norm of many;
        # the sums' errors are far below
        assert float((out[:m].double() - want).norm() / want.norm()) < (2.0 ** -8.5 if m * inner > 1000 else 2.0 ** -8)
        assert float(((out[:m].double() - want).abs() - 2.0 ** -8 * want.abs()).max()) < 1e-4
        assert bool((out[m:] == 3.0).all())
    kernels.check_status(a.device)


def test_large_gates_saturate():
    a = torch.tensor([[1.0] * 8, [-1.0] * 8], device=DEV).repeat(40, 1).bfloat16()
    w = torch.cat([torch.full((16, 8), 1e4, device=DEV), torch.ones(16, 8, device=DEV)]).bfloat16()
    for rule in ("gelu_new", "gelu", "swish"):
        out = torch.empty(80, 16, device=DEV).bfloat16()
        kernels.gated_tcgen05(a, w, out, m=80, activation=rule)
        want = paired((a.double() @ w.double().T)[:, :16], (a.double() @ w.double().T)[:, 16:], rule, 0.0)
        assert bool((out[0::2].double() - want[0::2]).abs().max() <= 2.0 ** -8 * want.abs().max()) and bool((out[1::2].float().abs() < 1e-30).all())


def test_gates_far_below_zero():
    # gates of which a large second factor leaves something: sigmoids down to 2^-128
    gates = torch.tensor([-20.0, -60.0, -85.0, -86.0, -87.0, -87.5, -88.0, -88.5], device=DEV)
    a = torch.ones(80, 8, device=DEV).bfloat16()
    w = torch.cat([gates[:, None] / 8.0 * torch.ones(8, device=DEV), torch.full((8, 8), 1e30, device=DEV)]).bfloat16()
    both, out = a.double() @ w.double().T, torch.empty(80, 8, device=DEV).bfloat16()
    kernels.gated_tcgen05(a, w, out, m=80, activation="swish")
    want = paired(both[:, :8], both[:, 8:], "swish", 0.0)
    # a rounding to bfloat16, and an exponential whose argument was rounded at 2^7: 2^-17 of it
    error = float(((out.double() - want) / want).abs().max())
    assert error < 2.0 ** -8
