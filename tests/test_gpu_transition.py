"""The forward in transition form (float32 storage; bf16 at D = 64): ragged chunk counts, both head dimensions, token-major and
grouped inputs, and decays too strong for the product form of a diagonal block.  Against the float64 recurrence."""
import pytest
import torch

import linearnexus_b200 as L
from linearnexus_b200 import _lib
from oracle import delta_rule_oracle as O

pytestmark = pytest.mark.gpu


def _truth(variant, i, rep=1):
    d = {k: None if t is None else t.double() for k, t in i.items()}
    q, k = (d[x].repeat_interleave(rep, dim=1) for x in ("q", "k"))
    if variant == "delta":
        return O.delta_rule_recurrent(q, k, d["v"], d["beta"], d["h0"], compute_dtype=torch.float64)
    f = O.gated_delta_rule_recurrent if variant == "gated" else O.kda_recurrent
    return f(q, k, d["v"], d["g"], d["beta"], initial_state=d["h0"], compute_dtype=torch.float64)


def _run(variant, i):
    if variant == "delta":
        return L.delta_rule_chunkwise(i["q"], i["k"], i["v"], i["beta"], i["h0"])
    f = L.gated_delta_rule_chunkwise if variant == "gated" else L.kda_chunkwise
    return f(i["q"], i["k"], i["v"], i["g"], i["beta"], initial_state=i["h0"])


def _err(a, b):
    return ((a.double().cpu() - b).abs().max() / b.abs().max()).item()


@pytest.mark.parametrize("variant", ["delta", "gated", "kda"])
@pytest.mark.parametrize("D,B,H,T,layout", [(64, 1, 2, 65, "bhtd"), (64, 2, 3, 200, "bthd"), (128, 1, 2, 127, "bthd"), (128, 2, 2, 193, "bhtd"),
                                            (64, 1, 40, 129, "bhtd"), (128, 3, 8, 130, "bhtd")])
def test_transition_form_float32(variant, D, B, H, T, layout):
    i = O.make_inputs(variant, B, H, T, D, D, seed=T + D, io_dtype=torch.float32, h0_std=0.1)
    c = {k: None if t is None else t.cuda() for k, t in i.items()}
    if layout == "bthd":
        c = {k: t if t is None or k == "h0" else t.transpose(1, 2).contiguous().transpose(1, 2) for k, t in c.items()}
    o, s = _run(variant, c)
    assert _lib.last_path() == "chunk_transition"
    ro, rs = _truth(variant, i)
    assert _err(o, ro) <= 5e-6 and _err(s, rs) <= 5e-6


def test_transition_form_strong_decay_and_grouped_heads():
    i = O.make_inputs("kda", 1, 4, 150, 64, 64, seed=9, io_dtype=torch.float32, h0_std=0.1)
    i["g"][:, :, 16:48] *= 400.0          # e^{-100} per token in places: far beyond the range of one block
    i["g"][:, :, 70, 3] = -1.0e4
    i["q"], i["k"] = i["q"][:, :2].contiguous(), i["k"][:, :2].contiguous()
    o, s = _run("kda", {k: None if t is None else t.cuda() for k, t in i.items()})
    assert _lib.last_path() == "chunk_transition" and torch.isfinite(o).all()
    ro, rs = _truth("kda", i, rep=2)
    assert _err(o, ro) <= 5e-6 and _err(s, rs) <= 5e-6


def test_transition_form_bf16_storage():
    i = O.make_inputs("gated", 2, 3, 140, 64, 64, seed=3, io_dtype=torch.bfloat16, h0_std=0.1)
    o, s = _run("gated", {k: None if t is None else t.cuda() for k, t in i.items()})
    assert _lib.last_path() == "chunk_transition" and o.dtype == torch.bfloat16
    ro, rs = _truth("gated", i)
    assert _err(o, ro) <= 5e-3 and _err(s, rs) <= 5e-6


@pytest.mark.parametrize("variant", ["delta", "gated", "kda"])
@pytest.mark.parametrize("B,H,Hq,T,layout", [(1, 2, 2, 64, "bhtd"), (1, 4, 2, 321, "bthd"), (2, 4, 4, 450, "bhtd"), (1, 20, 10, 200, "bthd"),
                                              (1, 7, 7, 64, "bhtd"), (1, 7, 7, 150, "bthd")])
def test_transition_form_bf16_tensor_shape(variant, B, H, Hq, T, layout):
    i = O.make_inputs(variant, B, H, T, 128, 128, seed=T, io_dtype=torch.bfloat16, h0_std=0.02)
    i["q"], i["k"] = i["q"][:, :Hq].contiguous(), i["k"][:, :Hq].contiguous()
    c = {k: None if t is None else t.cuda() for k, t in i.items()}
    if layout == "bthd":
        c = {k: t if t is None or k == "h0" else t.transpose(1, 2).contiguous().transpose(1, 2) for k, t in c.items()}
    kw = dict(initial_state=c["h0"], path="transition")
    if variant == "delta":
        o, s = L.delta_rule_chunkwise(c["q"], c["k"], c["v"], c["beta"], **kw)
    else:
        o, s = (L.gated_delta_rule_chunkwise if variant == "gated" else L.kda_chunkwise)(c["q"], c["k"], c["v"], c["g"], c["beta"], **kw)
    assert _lib.last_path() == "chunk_transition"
    ro, rs = _truth(variant, i, rep=H // Hq)
    assert _err(o, ro) <= 2e-2 and _err(s, rs) <= 2e-2
    if B * H <= 18 and T > 320 and variant != "kda":     # what AUTO takes for few sequences
        o2, s2 = _run(variant, c)
        assert _lib.last_path() == "chunk_transition" and torch.equal(o, o2) and torch.equal(s, s2)


@pytest.mark.parametrize("T", [40, 64, 150])
def test_per_channel_backward_with_strong_decay(T):
    """Blocks whose decay range exceeds the product form, in the pre-pass and in the local pass of the bf16 backward."""
    i = O.make_inputs("kda", 1, 2, T, 128, 128, seed=T, io_dtype=torch.bfloat16, h0_std=0.1)
    i["g"][:, :, 5:30] *= 300.0
    c = {k: None if t is None else t.cuda() for k, t in i.items()}
    from linearnexus_b200 import ops
    g = torch.Generator().manual_seed(1)
    do = torch.randn(i["v"].shape, generator=g).bfloat16()
    got = ops.chunk_backward("kda", c["q"], c["k"], c["v"], c["g"], c["beta"], do.cuda(), c["h0"])
    f = lambda t: t.float() if t.dtype == torch.bfloat16 else t
    ref = O.delta_rule_grads("kda", f(i["q"]), f(i["k"]), f(i["v"]), i["g"], i["beta"], i["h0"], f(do))
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):
        assert torch.isfinite(got[name]).all() and _err(got[name], ref[name].double()) <= 2e-2, name


@pytest.mark.parametrize("variant,D,tokens,decay", [("gated", 64, 8, -80.0), ("gated", 128, 8, -80.0), ("gated", 64, 1, -1.0e5),
                                                    ("gated", 128, 3, float("-inf")), ("kda", 64, 1, -40.0), ("kda", 128, 1, -40.0),
                                                    ("kda", 64, 2, float("-inf"))])
def test_transition_form_reset_inside_a_block(variant, D, tokens, decay):
    """Decays that drop the state at the head of every 16-row block: the weak decays behind them keep float32 precision (the
    bound is that of the other float32 cases), and an infinite log decay is a reset, not a NaN."""
    i = O.make_inputs(variant, 1, 2, 200, D, D, seed=3, io_dtype=torch.float32, h0_std=0.1)
    g = torch.where(torch.arange(200) % 16 < tokens, decay, -0.02)
    i["g"] = (g.expand(1, 2, 200) if variant == "gated" else g[:, None].expand(1, 2, 200, D)).contiguous()
    o, s = _run(variant, {k: t.cuda() for k, t in i.items()})
    assert _lib.last_path() == "chunk_transition"
    ro, rs = _truth(variant, i)
    assert _err(o, ro) <= 5e-6 and _err(s, rs) <= 5e-6


@pytest.mark.parametrize("variant,T", [("kda", 1100), ("gated", 400)])
def test_transition_form_bf16_wide_chunks(variant, T):
    """bf16: chunks that decay by more than 2^64 in some channel take the 16-row form, the others one product; a positive log decay too.  bf16
    operands and float32 sums: 2e-2 of the largest value, the budget of the other bf16 forwards."""
    inp = O.make_inputs(variant, 1, 3, T, 128, 128, seed=T, io_dtype=torch.bfloat16, h0_std=0.02)
    g = inp["g"]
    for h, x in enumerate((-44.3 / 64, -44.4 / 64, -300.0)):
        (g[:, h, 64:128, 5] if variant == "kda" else g[:, h, 64:128])[...] = x
    (g[:, 1, 200, 7] if variant == "kda" else g[:, 1, 200])[...] = 0.05
    cu = {k: (None if v is None else v.cuda()) for k, v in inp.items()}
    op, ref = (L.kda_chunkwise, O.kda_recurrent) if variant == "kda" else (L.gated_delta_rule_chunkwise, O.gated_delta_rule_recurrent)
    o, hT = op(cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], initial_state=cu["h0"], chunk_size=64)
    assert _lib.last_path() == "chunk_transition"
    L.check_device_status()
    ro, rS = ref(*(inp[x].double() for x in ("q", "k", "v", "g", "beta")), initial_state=inp["h0"].double(), compute_dtype=torch.float64)
    for got, want in ((o, ro), (hT, rS)):
        assert (got.double().cpu() - want).abs().max() <= 2e-2 * want.abs().max()


@pytest.mark.parametrize("H,T,path", [(13, 2117, "chunk_transition"), (18, 2117, "chunk_transition"), (19, 2117, "chunk_split_tcgen05"), (18, 1024, "chunk_split_tcgen05")])
def test_kda_route_by_sequences_and_chunks(H, T, path):
    """KDA in bf16: up to 18 sequences of more than 16 chunks take the transition form, past 32 chunks as before them; the others the two-kernel form.  The budget
    of the other bf16 forwards: 2e-2 of the largest value."""
    inp = O.make_inputs("kda", 1, H, T, 128, 128, seed=H, io_dtype=torch.bfloat16, h0_std=0.02)
    cu = {k: v.cuda() for k, v in inp.items()}
    o, hT = L.kda_chunkwise(cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], initial_state=cu["h0"], chunk_size=64)
    assert _lib.last_path() == path
    L.check_device_status()
    ro, rS = O.kda_recurrent(*(cu[x].double() for x in ("q", "k", "v", "g", "beta")), initial_state=cu["h0"].double(), compute_dtype=torch.float64)
    for got, want in ((o, ro), (hT, rS)):
        assert (got.double().cpu() - want.cpu()).abs().max() <= 2e-2 * want.cpu().abs().max()
