"""The native host path of the public calls (csrc/host_calls.cpp) against what the Python path does for the same arguments."""
import pytest
import torch

import linearnexus_b200 as L

pytestmark = pytest.mark.gpu


def _inputs(B=1, H=2, T=70, D=64, dtype=torch.float32, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")
    n = lambda *s: torch.nn.functional.normalize(f(*s), dim=-1).to(dtype)
    return dict(q=n(B, H, T, D), k=n(B, H, T, D), v=f(B, H, T, D).to(dtype), g=-f(B, H, T).abs() * 0.1, beta=torch.sigmoid(f(B, H, T)))


def _step():
    d = _inputs(64, 32, 1, 128)
    a = [x[:, :, 0].contiguous() for x in d.values()]
    S = torch.zeros(64, 32, 128, 128, device="cuda")
    return lambda: L.gated_delta_rule_step(*a, S)


def _chunk(grad=False, backward=False):
    d = _inputs(2, 16, 4096, 128, torch.bfloat16)
    a = [x.requires_grad_(grad) for x in d.values()]
    if not backward:
        return lambda: L.gated_delta_rule_chunkwise(*a)
    o, _ = L.gated_delta_rule_chunkwise(*a)
    d_o = torch.ones_like(o)
    return lambda: torch.autograd.grad(o, a, d_o, retain_graph=True)


def _scan():
    d = _inputs(8, 16, 2048, 64)
    w = -d["v"].abs()
    return lambda: L.dplr_delta_rule_recurrent(d["q"], d["k"], d["v"], d["q"], d["k"], w)


def _conv():
    x = torch.zeros(8, 4096, 2048, device="cuda")
    w = torch.zeros(4, 2048, device="cuda")
    return lambda: L.depthwise_conv1d_causal(x, w)


@pytest.mark.parametrize("make", [_step, _chunk, lambda: _chunk(True), lambda: _chunk(True, True), _scan, _conv],
                         ids=["step", "chunk", "train_fwd", "train_bwd", "scan", "conv"])
def test_an_allocation_that_does_not_fit_raises_what_torch_raises(make):
    """A limit on the caching allocator, not on the device: callers that shrink a batch catch torch.OutOfMemoryError."""
    L.check_device_status()   # (synchronises; also registers the device's status word, before which calls go the Python way)
    call = make()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (4 << 20)) / total)
    fill = []   # what the allocator still holds of freed blocks
    try:
        for size in (64 << 20, 16 << 20, 4 << 20):
            try:
                while True:
                    fill.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                pass
        with pytest.raises(torch.OutOfMemoryError):
            call()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        fill.clear()
    call()   # the same call goes through once there is room
    torch.cuda.synchronize()
