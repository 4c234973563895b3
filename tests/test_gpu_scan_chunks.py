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
                                         (1, 577, 1, 64, 64, 1), (1, 1100, 2, 64, 128, 1), (3, 129, 50, 64, 64, 5)])
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
