"""The native host path of the public calls (csrc/host_calls.cpp) against what the Python path does for the same arguments."""
import pytest
import torch

import linearnexus_b200 as L
from linearnexus_b200 import ops
from linearnexus_b200._lib import DeltaRuleError

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


class _Declines:
    """Stands in for the native functions: declines every call, as they do for what is not the plain case."""

    def __getattr__(self, name):
        return lambda *a: None


def _calls():
    """(name, argument tensors, call) of every public function with a native path, at small odd sizes."""
    g = torch.Generator(device="cuda").manual_seed(7)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")
    d = _inputs(2, 4, 70, 64)
    t = [x[:, :, 3].contiguous() for x in d.values()]
    p = [x[0].transpose(0, 1).contiguous() for x in d.values()]
    v4, lw = f(2, 70, 4, 64), -f(2, 4, 70, 64).abs()
    bm, cm = f(2, 70, 2, 64), f(2, 70, 2, 64)
    c = []
    add = lambda name, fn, *a, **kw: c.append((name, list(a), lambda *x: fn(*x, **kw)))
    add("gated_chunk", L.gated_delta_rule_chunkwise, *d.values())
    add("gated_chunk_view", L.gated_delta_rule_chunkwise, *(x.transpose(1, 2).contiguous().transpose(1, 2) for x in d.values()))
    add("delta_chunk", L.delta_rule_chunkwise, d["q"], d["k"], d["v"], d["beta"], f(2, 4, 64, 64))
    add("kda_chunk_bf16", L.kda_chunkwise, *(x.bfloat16() for x in (d["q"], d["k"], d["v"], lw)), d["beta"])
    add("gated_recurrent", L.gated_delta_rule_recurrent, *d.values())
    add("gated_step", L.gated_delta_rule_step, *t, f(2, 4, 64, 64))
    add("kda_step", L.kda_step, t[0], t[1], t[2], lw[:, :, 0].contiguous(), t[4], f(2, 4, 64, 64))
    add("packed", lambda q, k, v, g_, b: L.chunkwise_varlen("gated", q, k, v, g_, b, [0, 9, 70]), *p)
    add("conv", L.short_conv_silu, f(2, 9, 40), f(4, 40), f(40))
    add("gates", L.gated_deltanet_gates, f(2, 9, 4), f(2, 9, 4), f(4), f(4))
    add("kda_gate", lambda x, A: L.kda_gate(x, A, 8)[0], f(2, 9, 32), f(4))
    add("norm", L.rmsnorm_gated, d["v"], f(64), v4)
    add("rwkv7", L.dplr_delta_rule_recurrent, d["q"], d["k"], d["v"], -d["k"], d["k"], lw)
    add("rwkv6", L.rwkv6_recurrent, d["q"], d["k"], d["v"], lw, f(4, 64))
    add("ssd", lambda x, dt, A, b, c_, D: L.ssd_chunk_scan(x, dt, A, b, c_, D, n_groups=2), v4, f(2, 70, 4), -f(4).abs(), bm, cm, f(4))
    return c


def _flat(r):
    return [x for x in (r if isinstance(r, tuple) else (r,)) if x is not None]


def _check_all(run):
    for name, args, call in _calls():
        want = [x.clone() for x in _flat(call(*args))]
        got = _flat(run(args, call))
        assert len(got) == len(want), name
        for a, b in zip(got, want):
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b), name


def test_declined_calls_give_the_same_results(monkeypatch):
    L.check_device_status()
    want = [[x.clone() for x in _flat(call(*a))] for _, a, call in _calls()]
    monkeypatch.setattr(ops, "_host", _Declines())
    for (name, args, call), w in zip(_calls(), want):
        for a, b in zip(_flat(call(*args)), w):
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b), name


def test_native_calls_run_on_the_current_stream():
    """The inputs are filled on a side stream behind a delay; a launch on any other stream would read what was there before."""
    L.check_device_status()

    def run(args, call):
        late = [torch.full_like(x, 0.5) for x in args]
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            torch.cuda._sleep(2_000_000)
            for x, y in zip(late, args):
                x.copy_(y)
            r = call(*late)
        side.synchronize()
        return r
    _check_all(run)


def test_subclasses_and_strided_inputs_take_the_python_path():
    """Not the plain case: tensors of a subclass, and inputs neither contiguous nor token-major."""
    L.check_device_status()

    class Sub(torch.Tensor):
        pass
    _check_all(lambda args, call: tuple(x.as_subclass(torch.Tensor) for x in _flat(call(*(a.as_subclass(Sub) for a in args)))))

    def strided(args, call):
        wide = [torch.stack([x, torch.zeros_like(x)], dim=-1)[..., 0] for x in args]
        assert not any(x.is_contiguous() for x in wide if x.numel() > 1)
        return call(*wide)
    _check_all(strided)


def test_declined_calls_reach_the_python_errors():
    L.check_device_status()
    d = _inputs(1, 2, 70, 64)
    a = list(d.values())
    chunk, step = L.gated_delta_rule_chunkwise, L.gated_delta_rule_step
    one = [x[:, :, 0].contiguous() for x in a]
    state = torch.zeros(1, 2, 64, 64, device="cuda")
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        chunk(a[0].cpu(), *a[1:])
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        chunk(*(x.cpu() for x in a))
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        step(*one, state.cpu())
    with pytest.raises(ValueError, match="beta must be"):
        chunk(*a[:4], a[4][:, :1])
    with pytest.raises(ValueError, match="initial_state must be"):
        chunk(*a, initial_state=state[:, :1])
    with pytest.raises(ValueError, match="divisible by BC=16"):
        chunk(*a, chunk_size=24)
    with pytest.raises(ValueError, match="unknown chunk path"):
        chunk(*a, path="nothing")
    with pytest.raises(ValueError, match="state must be"):
        step(*one, state[:, :1])
    with pytest.raises(ValueError, match="contiguous float32 state cache"):
        step(*one, state.bfloat16(), inplace=True)
    with pytest.raises(ValueError, match="cu_seqlens must rise strictly"):
        L.chunkwise_varlen("gated", *(x[0].transpose(0, 1).contiguous() for x in a), [0, 70, 70])
    with pytest.raises(ValueError, match="weight must be"):
        L.short_conv_silu(torch.zeros(1, 5, 8, device="cuda"), torch.zeros(4, 9, device="cuda"))
    with pytest.raises(ValueError, match="u must be"):
        L.rwkv6_recurrent(a[0], a[1], a[2], a[0], torch.zeros(3, 64, device="cuda"))
    with pytest.raises(ValueError, match="n_groups"):
        L.ssd_chunk_scan(torch.zeros(1, 5, 4, 64, device="cuda"), torch.zeros(1, 5, 4, device="cuda"), torch.zeros(4, device="cuda"),
                         *(torch.zeros(1, 5, 2, 64, device="cuda"),) * 2, torch.zeros(4, device="cuda"), n_groups=3)
    with pytest.raises(DeltaRuleError, match="shape"):
        chunk(*(x[..., :63] if x.dim() == 4 else x for x in a))
