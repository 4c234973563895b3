"""Training through token-major views: read in place by the saving forward and the backward, same gradients as contiguous copies."""
import pytest
import torch

import linearnexus_b200 as L

pytestmark = pytest.mark.gpu
OPS = {"delta": L.delta_rule_chunkwise, "gated": L.gated_delta_rule_chunkwise, "kda": L.kda_chunkwise}


def _inputs(variant, B, T, Hq, H, D, dtype):
    gen = torch.Generator(device="cuda").manual_seed(T + H)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k = (torch.nn.functional.normalize(r(B, T, Hq, D), dim=-1).to(dtype) for _ in range(2))
    g = None if variant == "delta" else torch.nn.functional.logsigmoid(r(B, T, H, *([D] if variant == "kda" else [])) + 4)
    return [q, k, r(B, T, H, D).to(dtype), g, torch.sigmoid(r(B, T, H))]


@pytest.mark.parametrize("variant,T,Hq,H,D,dtype", [
    ("delta", 65, 2, 2, 128, torch.bfloat16), ("gated", 130, 2, 4, 128, torch.bfloat16), ("gated", 64, 3, 3, 64, torch.float32),
    ("kda", 63, 2, 2, 128, torch.bfloat16), ("kda", 200, 2, 4, 128, torch.bfloat16), ("kda", 2, 2, 2, 64, torch.bfloat16)])
@pytest.mark.parametrize("loss", ["output", "state", "both"])
def test_token_major_training_step(variant, T, Hq, H, D, dtype, loss):
    xs = _inputs(variant, 2, T, Hq, H, D, dtype)
    res = []
    for token_major in (True, False):
        leaves = [None if x is None else x.transpose(1, 2).detach() for x in xs]
        leaves = [None if x is None else (x if token_major else x.contiguous()).requires_grad_(True) for x in leaves]
        args = [x for x in leaves if x is not None]
        o, S = OPS[variant](*args, chunk_size=64)
        gen = torch.Generator(device="cuda").manual_seed(1)
        wo = torch.randn(o.shape, generator=gen, device="cuda").to(o.dtype)
        ws = torch.randn(S.shape, generator=gen, device="cuda")
        total = (0 if loss == "state" else (o * wo).sum()) + (0 if loss == "output" else (S * ws).sum())
        res.append([o.detach(), S.detach(), *torch.autograd.grad(total, args)])
    for a, b in zip(*res):
        assert a.shape == b.shape and a.dtype == b.dtype
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)
