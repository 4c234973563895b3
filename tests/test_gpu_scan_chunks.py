"""The chunk forms of the state scans (bf16 storage) at the edges of their tiles: ragged ends, the smallest length they
take, several value slices, grouped B and C, and the segmented (cluster) launch.  float32 state within 1e-4 and outputs
within one bf16 rounding of the float64 recurrence."""
import math

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
                                         (1, 4100, 1, 64, 64, 1), (5, 257, 32, 64, 128, 1),
                                         # both sides of the lines between whole sequences, two, four and eight segments (15, 33 and 74
                                         # clusters at once), and of those to the mma.sync form at N = 64
                                         (1, 641, 33, 64, 128, 1), (1, 700, 34, 64, 128, 1), (1, 900, 37, 128, 128, 1), (1, 900, 25, 192, 64, 1),
                                         (1, 2561, 15, 64, 128, 1), (1, 2600, 16, 64, 64, 1), (1, 768, 33, 64, 64, 1), (1, 769, 4, 64, 64, 1), (1, 960, 4, 64, 64, 1), (1, 961, 15, 64, 64, 1),
                                         (1, 961, 16, 64, 64, 1), (1, 2560, 5, 192, 64, 1), (1, 2561, 3, 64, 64, 1)])
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


@pytest.mark.parametrize("T,N", [(32, 128), (64, 64), (64, 128), (1000, 64)])
def test_ssd_non_finite_input_in_short_sequences(T, N):
    """The same in the mma.sync form: nothing before the token, and not the rest of its sixteen-token block either."""
    g = torch.Generator().manual_seed(T + N)
    f = lambda *s, scale=1.0: (torch.randn(*s, generator=g) * scale).cuda()
    x, dt, A, D = f(1, T, 2, 64).bfloat16(), f(1, T, 2), -torch.exp(f(2)), f(2)
    Bm, Cm = f(1, T, 1, N, scale=0.5).bfloat16(), f(1, T, 1, N, scale=0.5).bfloat16()
    y0, s0 = L.ssd_chunk_scan(x, dt, A, Bm, Cm, D)
    bad, gone = torch.zeros_like(y0, dtype=torch.bool), torch.zeros_like(s0, dtype=torch.bool)
    for n, t in enumerate(range(15, T, 53)):
        h, q = n % 2, (11 * n + 3) % 64
        x[0, t, h, q] = (float("inf"), float("nan"), -float("inf"))[n % 3]
        bad[0, t:, h, q] = True
        gone[0, h, q] = True
    x[0, T - 1, 0, 63], bad[0, T - 1, 0, 63], gone[0, 0, 63] = float("nan"), True, True
    y, s = L.ssd_chunk_scan(x, dt, A, Bm, Cm, D)
    assert torch.equal(torch.isfinite(y.float()), ~bad) and torch.equal(y[~bad], y0[~bad])
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


@pytest.mark.parametrize("first,second", [((2, 64), (0, 62)), ((66, 128), (64, 126)), ((70, 128), (0, 64))])
@pytest.mark.parametrize("most", [0.02, 0.2, 1.0])
def test_ssd_decay_weights_inside_a_chunk(first, second, most):
    """The weight of token j in the output of token i, e^{G_i - G_j} dt_j, to float32 precision: in every head two tokens whose weighted
    inputs cancel but for what float32 leaves of the second one's factor, so that the output is the error.  Tokens i from one
    half of a chunk of 128, j and k from the same or the other half; decays of up to ``most`` powers of two a token.

    Expected of each of the two weights, as relative variance.  Tokens of one 32-row block: one exponential of the rounded difference d
    (log2 units; two sums, each uniform over one unit in the last place of d, times ln 2; the exponential itself 6.0e-8 rms, measured
    over [-120, 0]) and two products (uniform, 2^-24 at most).  Other tokens: two factors of about one unit in the last place
    (2.6e-8 rms each) and three products.  512 heads: the rms over that expectation scatters by 3 %; bound five times that."""
    g = torch.Generator().manual_seed(first[0] + 1000 * second[1])
    Bt, H, T, N = 64, 8, 128, 128
    A = -(torch.rand(H, generator=g) * 0.9 + 0.1) * most * 4 * math.log(2)      # dt = 1/4
    x, Bm, Cm = torch.zeros(Bt, T, H, 64), torch.zeros(Bt, T, H, N), torch.zeros(Bt, T, H, N)
    pick = lambda r: torch.randint(*r, (Bt, H), generator=g)
    i, j, k = pick(first), pick(second), pick(second)
    j, k = torch.minimum(j, i - 1), torch.minimum(k, i - 1)
    k = torch.where(k == j, torch.where(j > 0, j - 1, j + 1), k)
    b, h = torch.arange(Bt)[:, None].expand(Bt, H), torch.arange(H)[None].expand(Bt, H)
    log_w = (A * 0.25).double()[None]
    wj, wk = torch.exp(log_w * (i - j)), torch.exp(log_w * (i - k))
    factor = -(wj / wk).float()
    hi = factor.bfloat16().float()
    mid = (factor - hi).bfloat16().float()
    lo = (factor - hi - mid).bfloat16().float()      # three bf16 terms are the float32 number
    Cm[b, i, h, 0] = Cm[b, i, h, 1] = Cm[b, i, h, 2] = 1
    Bm[b, j, h, 0] = 1
    Bm[b, k, h, 0], Bm[b, k, h, 1], Bm[b, k, h, 2] = hi, mid, lo
    x[b, j, h] = x[b, k, h] = 1
    c = lambda t: t.cuda()
    y, _ = L.ssd_chunk_scan(c(x).bfloat16(), c(torch.zeros(Bt, T, H)), c(A), c(Bm).bfloat16(), c(Cm).bfloat16(), c(torch.zeros(H)),
                            n_groups=H, dt_limit=(0.25, 0.25))
    err = (y.double().cpu()[b, i, h, 0] / 0.25 - (wj + (hi.double() + mid + lo) * wk)) / wj
    var = torch.zeros_like(err)
    for col in (j, k):
        d = (log_w * (i - col)).abs() / math.log(2)
        ulp = torch.exp2(torch.floor(torch.log2(d)) - 23)
        near = 2 * (ulp * math.log(2)) ** 2 / 12 + 6.0e-8 ** 2 + 2 * 2.0 ** -48 / 3
        var += torch.where(i // 32 == col // 32, near, torch.full_like(d, 2 * 2.6e-8 ** 2 + 3 * 2.0 ** -48 / 3))
    use = (i >= 2) & (k < i) & (k != j)
    assert (err ** 2 / var)[use].mean().sqrt().item() <= 1.15


@pytest.mark.parametrize("apart", [1, 40])
def test_ssd_weights_below_the_normal_range(apart):
    """A weight of 2^-130 between two tokens of a chunk still counts (as in the token recurrence): the input times 2^120 is 2^-10."""
    T, j = 128, 20
    x, Bm, Cm = torch.zeros(1, T, 1, 64), torch.zeros(1, T, 1, 128), torch.zeros(1, T, 1, 128)
    A = torch.tensor([-4 * 130 / apart * math.log(2)])
    x[0, j], Bm[0, j, 0, 0], Cm[0, j + apart, 0, 0] = 1, 2.0 ** 60, 2.0 ** 60
    c = lambda t: t.cuda()
    y, _ = L.ssd_chunk_scan(c(x).bfloat16(), c(torch.zeros(1, T, 1)), c(A), c(Bm).bfloat16(), c(Cm).bfloat16(), c(torch.zeros(1)), dt_limit=(0.25, 0.25))
    want = 0.25 * math.exp(A.double().item() * 0.25 * apart) * 2.0 ** 120
    assert (y[0, j + apart].double().cpu() / want - 1).abs().max().item() <= 5e-3


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
