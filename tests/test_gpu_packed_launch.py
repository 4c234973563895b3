"""One launch over a packed batch (tensor-core forwards): tails at every edge of a chunk, more sequences than one table
holds, and nothing of a neighbouring sequence reaching a tail.  Checked bit for bit against the op on each sequence."""
import pytest
import torch

import linearnexus_b200 as L
from linearnexus_b200 import _lib
from linearnexus_b200.synthetic import make_row

pytestmark = pytest.mark.gpu


def _alone(variant, x, lo, hi, h0):
    v = lambda t: None if t is None else t[lo:hi].unsqueeze(0).transpose(1, 2)
    op = {"delta": lambda: L.delta_rule_chunkwise(v(x["q"]), v(x["k"]), v(x["v"]), v(x["beta"]), h0),
          "gated": lambda: L.gated_delta_rule_chunkwise(v(x["q"]), v(x["k"]), v(x["v"]), v(x["g"]), v(x["beta"]), initial_state=h0),
          "kda": lambda: L.kda_chunkwise(v(x["q"]), v(x["k"]), v(x["v"]), v(x["g"]), v(x["beta"]), initial_state=h0)}
    o, s = op[variant]()
    return o[0].transpose(0, 1), s[0]


def _inputs(variant, total, H, seed):
    r = make_row(variant, H, total, 128, 128, seed, 0, io_dtype=torch.bfloat16)
    return {k: None if t is None else t[0].transpose(0, 1).contiguous().cuda() for k, t in r.items()}


@pytest.mark.parametrize("variant", ["delta", "gated", "kda"])
@pytest.mark.parametrize("lens,poison", [([1, 63, 64, 65, 7, 200, 128], False), ([70, 33, 64, 5, 129], True),
                                         ([3 + i % 5 for i in range(200)], False)])
def test_packed_launch(variant, lens, poison):
    H, n = 2, len(lens)
    cu = [sum(lens[:i]) for i in range(n + 1)]
    x = _inputs(variant, cu[-1], H, seed=5)
    if poison:   # every other sequence is all NaN: the ones before them must not notice
        for i in range(1, n, 2):
            for k in ("q", "k", "v"):
                x[k][cu[i]:cu[i + 1]] = float("nan")
    h0 = torch.randn(n, H, 128, 128, generator=torch.Generator().manual_seed(1)).cuda() * 0.02
    o, s = L.chunkwise_varlen(variant, x["q"], x["k"], x["v"], x["g"], x["beta"], cu, initial_state=h0)
    assert _lib.last_path() == ("chunk_split_tcgen05" if variant == "kda" else "chunk_tcgen05")
    L.check_device_status()
    for i in (range(0, n, 2) if poison else range(0, n, max(1, n // 12))):
        ro, rs = _alone(variant, x, cu[i], cu[i + 1], h0[i:i + 1])
        assert torch.equal(o[cu[i]:cu[i + 1]], ro) and torch.equal(s[i], rs), i
        assert torch.isfinite(ro.float()).all()


@pytest.mark.parametrize("native", [True, False])
def test_scratch_of_a_packed_batch_is_bounded(native):
    """14 sequences whose records would take 1.16 GB: at most 1 GiB is asked for, the batch goes in two launches, and the results are
    those of its halves (which fit) bit for bit."""
    n, T, H = 14, 4000, 16
    g = torch.Generator(device="cuda").manual_seed(0)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k, v = (f(n * T, H, 128).bfloat16() for _ in range(3))
    d = -f(n * T, H, 128).abs().mul_(0.05).bfloat16()
    beta = torch.sigmoid(f(n * T, H))
    if not native:   # another storage type of beta goes the Python way
        beta = beta.bfloat16()
    L.check_device_status()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    run = lambda a, b: L.chunkwise_varlen("kda", *(t[a * T:b * T] for t in (q, k, v, d, beta)), [i * T for i in range(b - a + 1)], out_dtype=torch.bfloat16)
    o, s = run(0, n)
    asked = torch.cuda.max_memory_allocated() - before
    results = o.numel() * 2 + s.numel() * 4 + (0 if native else beta.numel() * 4)
    assert asked <= results + (1 << 30) + (8 << 20)
    h = n // 2
    for a, b in ((0, h), (h, n)):
        ro, rs = run(a, b)
        assert torch.equal(o[a * T:b * T], ro) and torch.equal(s[a:b], rs)
    L.check_device_status()
