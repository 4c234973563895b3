"""The chunk forms of the state scans (bf16 storage) at the edges of their tiles: ragged ends, the smallest length they
take, several value slices, grouped B and C, and the segmented (cluster) launch.  float32 state within 1e-4 and outputs
within one bf16 rounding of the float64 recurrence."""
import pytest
import torch

import linearnexus_b200 as L
from oracle import linear_recurrences_oracle as R

pytestmark = pytest.mark.gpu


def _check(got, ref, tol):
    got, ref = got.double().cpu(), ref.double()
    assert ((got - ref).abs().max() / ref.abs().max().clamp_min(1e-30)).item() <= tol


@pytest.mark.parametrize("B,T,H,P,N,G", [(1, 32, 2, 64, 64, 1), (1, 63, 2, 64, 128, 2), (2, 65, 4, 128, 128, 2), (1, 200, 2, 64, 128, 1),
                                         (1, 577, 1, 64, 64, 1), (1, 1100, 2, 64, 128, 1), (3, 129, 50, 64, 64, 5),
                                         # tcgen05 form: one chunk, a whole one, one token more; four and eight segments, empty ones among
                                         # them; more CTAs than SMs; three value slices
                                         (1, 127, 2, 64, 64, 1), (2, 128, 2, 64, 128, 1), (1, 513, 3, 192, 128, 1), (1, 641, 2, 64, 128, 2),
                                         (1, 4100, 1, 64, 64, 1), (5, 257, 32, 64, 128, 1)])
def test_ssd_chunks(B, T, H, P, N, G):
    g = torch.Generator().manual_seed(T)
    f = lambda *s, scale=1.0: torch.randn(*s, generator=g) * scale
    bf = lambda t: t.bfloat16()
    x, dt, A = bf(f(B, T, H, P)), f(B, T, H, scale=0.5), -torch.exp(f(H, scale=0.5))
    Bm, Cm, D, bias, h0 = bf(f(B, T, G, N, scale=0.5)), bf(f(B, T, G, N, scale=0.5)), f(H), f(H, scale=0.3), f(B, H, P, N, scale=0.1)
    c = lambda t: t.cuda()
    kw = dict(n_groups=G, dt_limit=(0.001, 5.0))
    y, s = L.ssd_chunk_scan(c(x), c(dt), c(A), c(Bm), c(Cm), c(D), ssm_state=c(h0), dt_bias=c(bias), **kw)
    d = lambda t: t.double()
    ry, rs = R.ssd_chunk_scan(d(x), d(dt), d(A), d(Bm), d(Cm), d(D), ssm_state=d(h0), dt_bias=d(bias), compute_dtype=torch.float64,
                              chunk_size=64, **kw)
    _check(s, rs, 1e-5)
    _check(y, ry, 5e-3)


@pytest.mark.parametrize("N", [64, 128])
def test_ssd_non_finite_input(N):
    """An infinity or NaN in x reaches the outputs of its own column from its token on, and the state, and nothing before it."""
    g = torch.Generator().manual_seed(N)
    f = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).cuda()
    x, dt, A, D = f(1, 300, 2, 64).bfloat16(), f(1, 300, 2), -torch.exp(f(2)), f(2)
    Bm, Cm = f(1, 300, 1, N, scale=0.5).bfloat16(), f(1, 300, 1, N, scale=0.5).bfloat16()
    y0, s0 = L.ssd_chunk_scan(x, dt, A, Bm, Cm, D)
    x[0, 70, 1, 5], x[0, 200, 1, 6] = float("inf"), float("nan")
    y, s = L.ssd_chunk_scan(x, dt, A, Bm, Cm, D)
    bad = torch.zeros_like(y, dtype=torch.bool)
    bad[0, 70:, 1, 5] = bad[0, 200:, 1, 6] = True
    assert torch.equal(torch.isfinite(y.float()), ~bad) and torch.equal(y[~bad], y0[~bad])
    gone = torch.zeros_like(s, dtype=torch.bool)
    gone[0, 1, 5:7] = True
    assert torch.equal(torch.isfinite(s), ~gone) and torch.equal(s[~gone], s0[~gone])


@pytest.mark.parametrize("B,T,H,N", [(1, 4100, 2, 128), (1, 1100, 4, 128), (1, 1100, 4, 64), (2, 1000, 45, 128)])
def test_ssd_non_finite_input_in_every_chunk(B, T, H, N):
    """One non-finite x in each chunk of every segment (eight, four, four and one of them), each in a column of its own: a chunk's notes
    must not be taken for those of a neighbour that uses the same stage."""
    g = torch.Generator().manual_seed(T + N)
    f = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).cuda()
    x, dt, A, D = f(B, T, H, 64).bfloat16(), f(B, T, H), -torch.exp(f(H)), f(H)
    Bm, Cm = f(B, T, 1, N, scale=0.5).bfloat16(), f(B, T, 1, N, scale=0.5).bfloat16()
    y0, s0 = L.ssd_chunk_scan(x, dt, A, Bm, Cm, D)
    bad, gone = torch.zeros_like(y0, dtype=torch.bool), torch.zeros_like(s0, dtype=torch.bool)
    for c in range(0, T, 128):
        n = c // 128
        t, h, q = min(T - 1, c + 37 * n % 128), n % H, (5 * n + 3) % 64
        x[:, t, h, q] = (float("inf"), float("nan"), -float("inf"))[n % 3]
        bad[:, t:, h, q] = True
        gone[:, h, q] = True
    y, s = L.ssd_chunk_scan(x, dt, A, Bm, Cm, D)
    assert torch.equal(torch.isfinite(y.float()), ~bad) and torch.equal(y[~bad], y0[~bad])
    assert torch.equal(torch.isfinite(s), ~gone) and torch.equal(s[~gone], s0[~gone])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,H,T,V,layout", [(1, 2, 9, 64, "bhtd"), (2, 3, 31, 128, "bthd"), (1, 2, 130, 64, "bhtd"), (1, 1, 203, 192, "bhtd")])
def test_rwkv_blocks(dtype, B, H, T, V, layout):
    """Eight tokens per step of the state: tails of every length, several value slices, strong and vanishing decays."""
    g = torch.Generator().manual_seed(T)
    f = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).to(dtype)
    kk = torch.nn.functional.normalize(torch.randn(B, H, T, 64, generator=g), dim=-1)
    q, k, v = f(B, H, T, 64), f(B, H, T, 64, scale=0.5), f(B, H, T, V)
    a, b = (-kk).to(dtype), (kk * torch.sigmoid(torch.randn(B, H, T, 64, generator=g))).to(dtype)
    gk, u, h0 = -torch.exp(f(B, H, T, 64) - 1.0), torch.randn(H, 64, generator=g) * 0.5, torch.randn(B, H, 64, V, generator=g) * 0.1
    gk[:, :, T // 2] = -60.0
    gk[:, :, T // 3] = 0.0
    gk = gk.to(dtype)
    dev = lambda t: t.cuda() if layout == "bhtd" else t.transpose(1, 2).contiguous().cuda().transpose(1, 2)
    d = lambda t: t.double()
    tol = 5e-3 if dtype == torch.bfloat16 else 5e-6
    o, s = L.dplr_delta_rule_recurrent(*(dev(t) for t in (q, k, v, a, b, gk)), scale=0.125, initial_state=h0.cuda())
    ro, rs = R.dplr_delta_rule_recurrent(*(d(t) for t in (q, k, v, a, b, gk)), scale=0.125, initial_state=d(h0), compute_dtype=torch.float64)
    _check(s, rs, 5e-6)
    _check(o, ro, tol)
    w = (-torch.randn(B, H, T, 64, generator=g).abs() - 0.5).to(dtype)
    w[:, :, T // 2] = 5.0
    o, s = L.rwkv6_recurrent(*(dev(t) for t in (q, k, v, w)), u.cuda(), scale=0.125, initial_state=h0.cuda())
    ro, rs = R.rwkv6_recurrent(*(d(t) for t in (q, k, v, w, u)), scale=0.125, initial_state=d(h0), compute_dtype=torch.float64)
    _check(s, rs, 5e-6)
    _check(o, ro, tol)


@pytest.mark.parametrize("B,T,H,N,first,A", [(1, 64, 2, 128, 32, -16.0), (1, 200, 2, 64, 1, -16.0), (2, 130, 80, 128, 20, -4.0),
                                             (1, 1100, 2, 128, 32, -16.0), (1, 200, 2, 64, 5, -1.0e6)])
def test_ssd_reset_then_accumulate(B, T, H, N, first, A):
    """A strong decay in the first tokens of every chunk (the state is dropped), weak ones behind it: the chunk form has to keep the
    weak decays to float32 precision, as the token recurrence does.  Bound: dt' = softplus(dt) in float32 is within 3e-7 of 64 bits
    and enters a weight as factor and as exponent (|A dt'| <= 0.32 a token, e-folding after a few), the sums and products add a few
    2^-24 each; 1.5e-6 of the state's largest entry.  A float32 running sum over the chunk misses it by two orders."""
    g = torch.Generator().manual_seed(T)
    f = lambda *s, scale=1.0: torch.randn(*s, generator=g) * scale
    bf = lambda t: t.bfloat16()
    x, Bm, Cm, D = bf(f(B, T, H, 64)), bf(f(B, T, 1, N, scale=0.5)), bf(f(B, T, 1, N, scale=0.5)), f(H)
    weak = min(0.02, 0.32 / -A)
    dt = torch.where((torch.arange(T) % 64 < first)[None, :, None], torch.tensor(5.0), torch.tensor(weak).expm1().log()).expand(B, T, H)
    dt = (dt + f(B, T, H, scale=0.01)).contiguous()
    Ah, h0 = torch.full((H,), A), f(B, H, 64, N)
    c, d = (lambda t: t.cuda()), (lambda t: t.double())
    y, s = L.ssd_chunk_scan(c(x), c(dt), c(Ah), c(Bm), c(Cm), c(D), ssm_state=c(h0))
    ry, rs = R.ssd_token_recurrence(d(x), d(dt), d(Ah), d(Bm), d(Cm), d(D), ssm_state=d(h0))
    _check(s, rs, 1.5e-6)
    _check(y, ry, 5e-3)


@pytest.mark.parametrize("T", [9, 39, 40, 41])
def test_rwkv_more_sequences_than_sms(T):
    """Two waves of slices, on both sides of the line between the token recurrence and the blocks (20 tokens a wave)."""
    g = torch.Generator().manual_seed(T)
    f = lambda *s: torch.randn(*s, generator=g)
    kk = torch.nn.functional.normalize(f(1, 150, T, 64), dim=-1)
    x = (f(1, 150, T, 64), f(1, 150, T, 64) * 0.5, f(1, 150, T, 64), -kk, kk * torch.sigmoid(f(1, 150, T, 64)), -torch.exp(f(1, 150, T, 64) - 1.0))
    o, s = L.dplr_delta_rule_recurrent(*(t.cuda() for t in x), scale=0.125)
    ro, rs = R.dplr_delta_rule_recurrent(*(t.double() for t in x), scale=0.125, compute_dtype=torch.float64)
    _check(o, ro, 5e-6)
    _check(s, rs, 5e-6)
