"""The recurrences' chunks on tensor cores at the ends of the numbers' range.  Values that have no parts: infinities, and 32-bit numbers that
bfloat16 rounds to one, against the chunks' formulas in 64 bits, token by token in the order of time: what is a number there is one here, what
is an infinity has its sign, and no token's result depends on a later token.  And x sigmoid(x) far below zero."""
import pytest
import torch

from burn_transformers_b200 import kernels

pytestmark = pytest.mark.gpu
DEV, F64 = "cuda", torch.float64
CHUNK, LENGTHS, HEADS = 64, [70, 300], 16


def step(lengths):
    starts = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    return starts, ints(starts), ints(list(range(len(lengths), 0, -1)))


def outer(k, v):
    return k[:, :, None] * v[:, None, :]


def dot(q, m):      # sum over the key channels, without a library product (whose padding would meet the infinities)
    return (q[:, :, None] * m).sum(1)


def same(got, want, size):
    """Equal kinds everywhere; where `want` is a number, within what sums of some hundred 32-bit terms of total `size` may lose."""
    got, inf = got.to(F64).reshape(want.shape), torch.isinf(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[inf], want[inf])
    ok = torch.isfinite(want) & torch.isfinite(size)
    assert float(((got - want).abs()[ok] / size[ok].clamp_min(1e-300)).max()) < 256 * 2.0 ** -23


def spoil(rows, lo, v, kind, dim, vdim):
    """Puts the numbers in question into the values (at offset v) of the sequence whose rows begin at lo."""
    if kind == "infinite":
        rows[lo + 21, v + 2 * vdim + 5] = float("inf")
        rows[lo + 100, v + 3 * vdim] = float("-inf")
        rows[lo + 5, v + 4 * vdim + vdim - 1] = float("nan")
    else:
        rows[lo + 30, v + 2 * vdim + 5] = 3.4e38
        rows[lo + 77, v + 3 * vdim] = -3.4e38


KINDS = [(torch.bfloat16, "infinite"), (torch.float32, "infinite"), (torch.float32, "largest")]


@pytest.mark.parametrize("dim, vdim", [(16, 24), (64, 64), (128, 72)])
@pytest.mark.parametrize("dtype, kind", KINDS)
@pytest.mark.parametrize("activation", ["swish", None])
def test_decayed_chunks(dim, vdim, dtype, kind, activation):
    torch.manual_seed(dim)
    starts, seq_start, slots = step(LENGTHS)
    n, wide = starts[-1], HEADS * (2 * dim + vdim)
    rows = torch.randn(n, wide, device=DEV) * (1e-3 if kind == "largest" else 1.0)
    spoil(rows, starts[1], 2 * HEADS * dim, kind, dim, vdim)
    if activation and kind == "infinite":
        rows.nan_to_num_(nan=float("nan"), posinf=float("inf"), neginf=float("inf"))      # (x sigmoid(x) of minus infinity is no number)
    proj, decay = rows.to(dtype), torch.rand(HEADS, device=DEV) * 0.2 + 0.8
    state = torch.randn(3, HEADS, dim, vdim, device=DEV)
    first, out = state.clone(), torch.empty(n, HEADS * vdim, device=DEV)
    scratch = torch.empty(kernels.lightning_chunked_scratch_floats(2, max(LENGTHS), HEADS, dim, vdim), device=DEV)
    kernels.lightning_scan(proj, 0, HEADS * dim, 2 * HEADS * dim, state, slots, seq_start, decay, out, n_seqs=2, n_heads=HEADS, dim=dim,
                           vdim=vdim, max_new=max(LENGTHS), scratch=scratch, activation=activation)
    x, lam = proj.to(F64), decay.to(F64)[:, None]
    x = x * torch.sigmoid(x) if activation else x
    for i in range(2):
        S = first[2 - i].to(F64)
        T = S.abs()      # the same with every number's size
        want, size = [], []
        for lo in range(starts[i], starts[i + 1], CHUNK):
            hi = min(lo + CHUNK, starts[i + 1])
            q, k, v = (x[lo:hi, a:a + HEADS * d].view(hi - lo, HEADS, d) for a, d in ((0, dim), (HEADS * dim, dim), (2 * HEADS * dim, vdim)))
            for t in range(hi - lo):
                o, u = lam ** (t + 1) * dot(q[t], S), lam ** (t + 1) * dot(q[t].abs(), T)
                for s in range(t + 1):
                    o = o + lam ** (t - s) * (q[t] * k[s]).sum(-1, keepdim=True) * v[s]
                    u = u + lam ** (t - s) * (q[t] * k[s]).abs().sum(-1, keepdim=True) * v[s].abs()
                want.append(o)
                size.append(u)
            fall = lam[:, :, None] ** (hi - lo)
            S, T = fall * S, fall * T
            for s in range(hi - lo):
                f = lam[:, :, None] ** (hi - lo - 1 - s)
                S, T = S + f * outer(k[s], v[s]), T + f * outer(k[s], v[s]).abs()
        same(out[starts[i]:starts[i + 1]], torch.stack(want), torch.stack(size))
        same(state[2 - i], S, T)


@pytest.mark.parametrize("dim, vdim", [(16, 24), (64, 64), (128, 72)])
@pytest.mark.parametrize("dtype, kind", KINDS + [(torch.bfloat16, "key"), (torch.float32, "key")])
def test_memory_chunks(dim, vdim, dtype, kind):
    torch.manual_seed(dim)
    starts, seq_start, slots = step(LENGTHS)
    n, wide = starts[-1], HEADS * (2 * dim + vdim)
    rows = torch.randn(n, wide + 2 * HEADS, device=DEV)
    if kind == "largest":
        rows[:, :wide] *= 1e-3
    if kind == "key":
        rows[starts[1] + 37, HEADS * dim + 6 * dim + 3] = float("inf")
    else:
        spoil(rows, starts[1], 2 * HEADS * dim, kind, dim, vdim)
    proj = rows.to(dtype)
    bias_i, bias_f = torch.randn(HEADS, device=DEV) - 1.0, torch.rand(HEADS, device=DEV) * 2.0 + 2.0
    s, nn, m = (torch.randn(3, HEADS, *d, device=DEV) for d in ((dim, vdim), (dim,), ()))
    before, out = tuple(t.clone() for t in (s, nn, m)), torch.empty(n, HEADS * vdim, device=DEV)
    scratch = torch.empty(kernels.mlstm_chunked_scratch_floats(n, 2, max(LENGTHS), HEADS, dim, vdim), device=DEV)
    kernels.mlstm_scan(proj, (0, HEADS * dim, 2 * HEADS * dim, wide, wide + HEADS), bias_i, bias_f, 15.0, dim ** -0.5, s, nn, m, slots,
                       seq_start, out, n_seqs=2, n_heads=HEADS, dim=dim, vdim=vdim, max_new=max(LENGTHS), scratch=scratch)
    x = proj.to(F64)
    a = 15.0 * torch.tanh((x[:, wide:wide + HEADS] + bias_i.to(F64)) / 15.0)
    b = torch.nn.functional.logsigmoid(15.0 * torch.tanh((x[:, wide + HEADS:] + bias_f.to(F64)) / 15.0))
    for i in range(2):
        S, N, top = (t[2 - i].to(F64) for t in before)
        T, M = S.abs(), N.abs()
        want, size = [], []
        for lo in range(starts[i], starts[i + 1], CHUNK):
            hi = min(lo + CHUNK, starts[i + 1])
            q, k, v = (x[lo:hi, c:c + HEADS * d].view(hi - lo, HEADS, d) for c, d in ((0, dim), (HEADS * dim, dim), (2 * HEADS * dim, vdim)))
            ca, ab, m_in, tops = torch.cumsum(b[lo:hi], 0), a[lo:hi], top, []
            for t in range(hi - lo):
                top = torch.maximum(b[lo + t] + top, ab[t])
                tops.append(top)
                f, qt = torch.exp(ca[t] + m_in - top)[:, None], q[t] * dim ** -0.5
                num, den = f * dot(qt, S), f * (qt * N).sum(-1, keepdim=True)
                num_s, den_s = f * dot(qt.abs(), T), f * (qt.abs() * M).sum(-1, keepdim=True)
                for r in range(t + 1):
                    w = torch.exp(ca[t] - ca[r] + ab[r] - top)[:, None]
                    num, den = num + w * (qt * k[r]).sum(-1, keepdim=True) * v[r], den + w * (qt * k[r]).sum(-1, keepdim=True)
                    grown = w * (qt * k[r]).abs().sum(-1, keepdim=True)
                    num_s, den_s = num_s + grown * v[r].abs(), den_s + grown
                by = torch.fmax(den.abs(), torch.exp(-top)[:, None]) + 1e-6
                want.append(num / by)
                size.append(num_s / by + (num / by).abs() * den_s / by)
            keep = torch.exp(ca[-1] + m_in - top)
            S, T, N, M = keep[:, None, None] * S, keep[:, None, None] * T, keep[:, None] * N, keep[:, None] * M
            for r in range(hi - lo):
                w = torch.exp(ca[-1] - ca[r] + ab[r] - top)[:, None]
                S, T = S + outer(w * k[r], v[r]), T + outer(w * k[r], v[r]).abs()
                N, M = N + w * k[r], M + (w * k[r]).abs()
        # (a weight is e to a 32-bit sum of up to 64 log gates: an error of some units in its exponent of up to about 100)
        same(out[starts[i]:starts[i + 1]], torch.stack(want), 8.0 * torch.stack(size))
        same(s[2 - i], S, 8.0 * T)
        same(nn[2 - i], N, 8.0 * M)


@pytest.mark.parametrize("dim, vdim", [(32, 24), (64, 64), (48, 72)])
@pytest.mark.parametrize("dtype, kind", KINDS)
def test_gated_chunks(dim, vdim, dtype, kind):
    torch.manual_seed(dim)
    starts, seq_start, slots = step(LENGTHS)
    n, wide = starts[-1], HEADS * (2 * dim + vdim)
    rows = torch.randn(n, wide, device=DEV) * (1e-3 if kind == "largest" else 1.0)
    spoil(rows, starts[1], 2 * HEADS * dim, kind, dim, vdim)
    proj, dt = rows.to(dtype), torch.rand(n, HEADS * dim, device=DEV)
    state = torch.randn(3, HEADS, dim, vdim, device=DEV)
    first, out = state.clone(), torch.empty(n, HEADS * vdim, device=DEV)
    scratch = torch.empty(kernels.gla_chunked_scratch_floats(n, 2, max(LENGTHS), HEADS, dim, vdim), device=DEV)
    kernels.gla_scan(proj, 0, HEADS * dim, 2 * HEADS * dim, dim ** -0.5, dt, -0.25, state, slots, seq_start, out, n_seqs=2, n_heads=HEADS,
                     dim=dim, vdim=vdim, max_new=max(LENGTHS), scratch=scratch)
    x, log_a = proj.to(F64), -0.25 * dt.to(F64).view(n, HEADS, dim)
    for i in range(2):
        S = first[2 - i].to(F64)
        T = S.abs()
        want, size = [], []
        for lo in range(starts[i], starts[i + 1], CHUNK):
            hi = min(lo + CHUNK, starts[i + 1])
            q, k, v = (x[lo:hi, a:a + HEADS * d].view(hi - lo, HEADS, d) for a, d in ((0, dim), (HEADS * dim, dim), (2 * HEADS * dim, vdim)))
            b = torch.cumsum(log_a[lo:hi], 0)
            for t in range(hi - lo):
                qt = q[t] * dim ** -0.5
                o, u = dot(qt * torch.exp(b[t]), S), dot(qt.abs() * torch.exp(b[t]), T)
                for s in range(t + 1):
                    w = qt * k[s] * torch.exp(b[t] - b[s])
                    o, u = o + w.sum(-1, keepdim=True) * v[s], u + w.abs().sum(-1, keepdim=True) * v[s].abs()
                want.append(o)
                size.append(u)
            S, T = torch.exp(b[-1])[:, :, None] * S, torch.exp(b[-1])[:, :, None] * T
            for s in range(hi - lo):
                f = torch.exp(b[-1] - b[s])
                S, T = S + outer(f * k[s], v[s]), T + outer(f * k[s], v[s]).abs()
        same(out[starts[i]:starts[i + 1]], torch.stack(want), 4.0 * torch.stack(size))      # (a decay of up to 64 times 1/4 in its exponent)
        same(state[2 - i], S, 4.0 * T)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_feature_far_below_zero(dtype):
    heads, dim, n = 16, 16, 640
    values = torch.tensor([-20.0, -60.0, -86.5, -87.5, -88.5, -95.0, -104.0, -1e10, -1e30, -3e38], device=DEV).to(dtype)
    proj = torch.full((n, 3 * heads * dim), 1e4, device=DEV, dtype=dtype)
    proj[:, 2 * heads * dim:] = values.repeat(n * heads * dim // len(values)).view(n, -1)
    state, out = torch.zeros(1, heads, dim, dim, device=DEV), torch.empty(n, heads * dim, device=DEV)
    scratch = torch.empty(kernels.lightning_chunked_scratch_floats(1, n, heads, dim, dim), device=DEV)
    ints = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)  # noqa: E731
    kernels.lightning_scan(proj, 0, heads * dim, 2 * heads * dim, state, ints(0), ints(0, n), torch.zeros(heads, device=DEV), out, n_seqs=1,
                           n_heads=heads, dim=dim, vdim=dim, max_new=n, scratch=scratch)
    v = proj[:, 2 * heads * dim:].to(F64)
    want = dim * proj[0, 0].to(F64) ** 2 * v / (1.0 + torch.exp(-v))      # (a decay of zero: a token sees itself alone)
    # (below 2^-110 a number's parts have fewer bits: the last of bfloat16's numbers is 2^-133)
    error = float(((out.to(F64) - want).abs() / (1e-5 * want.abs() + dim * 1e8 * 2.0 ** -132)).max())
    assert error < 1.0
