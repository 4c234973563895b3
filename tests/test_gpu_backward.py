"""GPU parity of the backward (dq, dk, dv, dbeta, dg, dh0) against autograd of the float64 oracle,
which is what jax.grad of the reference functions computes."""
import pytest
import torch

import linearnexus_b200 as L
from linearnexus_b200 import ops
from oracle import delta_rule_oracle as O

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return ((a - b).abs().max() / b.abs().max().clamp_min(1e-30)).item()


def _check(variant, B, H, T, K, V, C, io=torch.float32, tol=2e-4, h0_std=0.1, with_dhT=True):
    inp = O.make_inputs(variant, B, H, T, K, V, seed=T + K + C, io_dtype=io, h0_std=h0_std)
    if io == torch.float32:
        inp["q"] = inp["q"] * 1.3
        inp["k"] = inp["k"] * 0.7
    gen = torch.Generator().manual_seed(5)
    do = torch.randn(B, H, T, V, generator=gen).to(io)
    dhT = torch.randn(B, H, K, V, generator=gen) * 0.1 if with_dhT else None
    l2 = variant != "delta"
    f = lambda x: None if x is None else x.float() if x.dtype == torch.bfloat16 else x
    ref = O.delta_rule_grads(variant, f(inp["q"]), f(inp["k"]), f(inp["v"]), inp["g"], inp["beta"], inp["h0"], f(do), dhT,
                             use_qk_l2norm=l2)
    cu = lambda x: None if x is None else x.cuda()
    got = ops.chunk_backward(variant, cu(inp["q"]), cu(inp["k"]), cu(inp["v"]), cu(inp["g"]), cu(inp["beta"]), cu(do),
                             initial_state=cu(inp["h0"]), d_final_state=cu(dhT), chunk_size=C, use_qk_l2norm=l2)
    torch.cuda.synchronize()
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):
        if ref[name] is None:
            assert got[name] is None
            continue
        assert got[name].shape == ref[name].shape, name
        err = _rel(got[name], ref[name])
        assert err <= tol, f"{variant} {name}: rel err {err}"
    return got


@pytest.mark.parametrize("variant", ["delta", "gated", "kda"])
@pytest.mark.parametrize("shape", [(1, 2, 64, 32, 32, 64), (2, 2, 100, 16, 48, 32), (1, 1, 130, 64, 64, 64), (1, 2, 40, 128, 128, 16)])
def test_backward_fp32(variant, shape):
    _check(variant, *shape)


def test_backward_golden_fixture(golden):
    for name in ("delta", "gated", "kda"):
        G = lambda key: torch.from_numpy(golden[f"{name}.{key}"]).cuda() if f"{name}.{key}" in golden.files else None
        got = ops.chunk_backward(name, G("q"), G("k"), G("v"), G("g"), G("beta"), G("do"), initial_state=G("h0"),
                                 d_final_state=G("dhT"), chunk_size=int(golden[f"{name}.chunk"]), use_qk_l2norm=(name != "delta"))
        for key in ("dq", "dk", "dv", "dg", "dbeta", "dh0"):
            if G(key) is not None:
                assert _rel(got[key], G(key)) <= 2e-4, (name, key)


def test_backward_bf16_headline_head_size():
    """bf16 q,k,v,do with fp32 accumulation at d_k = d_v = 128, chunk 64 (the training configuration's head)."""
    got = _check("gated", 1, 2, 256, 128, 128, 64, io=torch.bfloat16, tol=2e-2, h0_std=0.02)
    assert got["dq"].dtype == torch.bfloat16 and got["dg"].dtype == torch.float32


def test_autograd_through_the_op():
    inp = O.make_inputs("gated", 1, 2, 96, 32, 32, seed=9, h0_std=0.1)
    leaf = {k_: (None if v_ is None else v_.cuda().requires_grad_(True)) for k_, v_ in inp.items()}
    o, hT = L.gated_delta_rule_chunkwise(leaf["q"], leaf["k"], leaf["v"], leaf["g"], leaf["beta"], initial_state=leaf["h0"],
                                         chunk_size=32)
    gen = torch.Generator().manual_seed(1)
    do = torch.randn(o.shape, generator=gen)
    dhT = torch.randn(hT.shape, generator=gen) * 0.1
    ((o * do.cuda()).sum() + (hT * dhT.cuda()).sum()).backward()
    ref = O.delta_rule_grads("gated", inp["q"], inp["k"], inp["v"], inp["g"], inp["beta"], inp["h0"], do, dhT)
    for name, key in (("q", "dq"), ("k", "dk"), ("v", "dv"), ("g", "dg"), ("beta", "dbeta"), ("h0", "dh0")):
        assert _rel(leaf[name].grad, ref[key]) <= 2e-4, key


@pytest.mark.parametrize("variant,io,K,tol", [("gated", torch.bfloat16, 128, 2e-2), ("delta", torch.bfloat16, 128, 2e-2),
                                              ("kda", torch.bfloat16, 128, 2e-2), ("gated", torch.float32, 32, 2e-4),
                                              ("kda", torch.float32, 16, 2e-4)])
def test_saving_forward_then_saved_backward(variant, io, K, tol):
    """One forward per training step: chunk_forward_saving returns the forward's results plus the per-chunk states;
    chunk_backward(saved=...) must give the gradients of the recomputing backward (and of the float64 oracle)."""
    from linearnexus_b200 import _lib
    B, H, T, C = 1, 2, 200, 64 if K == 128 else 32
    inp = O.make_inputs(variant, B, H, T, K, K, seed=21, io_dtype=io, h0_std=0.02)
    gen = torch.Generator().manual_seed(6)
    do = torch.randn(B, H, T, K, generator=gen).to(io)
    l2 = variant != "delta"
    cu = {k_: (None if v_ is None else v_.cuda()) for k_, v_ in inp.items()}
    o, hT, saved = ops.chunk_forward_saving(variant, cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], cu["h0"],
                                            chunk_size=C, use_qk_l2norm=l2)
    assert _lib.last_path() == "fwd_saving"
    # same forward results as the plain op (same kernels for gated/delta; KDA's default op is the same two-kernel path)
    if variant == "delta":
        o2, hT2 = L.delta_rule_chunkwise(cu["q"], cu["k"], cu["v"], cu["beta"], cu["h0"], chunk_size=C)
    elif variant == "gated":
        o2, hT2 = L.gated_delta_rule_chunkwise(cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], initial_state=cu["h0"], chunk_size=C)
    else:
        o2, hT2 = L.kda_chunkwise(cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], initial_state=cu["h0"], chunk_size=C)
    assert o.dtype == o2.dtype and torch.equal(o, o2) and torch.equal(hT, hT2)
    got = ops.chunk_backward(variant, cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], do.cuda(), initial_state=cu["h0"],
                             chunk_size=C, use_qk_l2norm=l2, saved=saved)
    assert _lib.last_path() == "bwd_saved"
    again = ops.chunk_backward(variant, cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], do.cuda(), initial_state=cu["h0"],
                               chunk_size=C, use_qk_l2norm=l2)
    f = lambda x: None if x is None else x.float() if x.dtype == torch.bfloat16 else x
    ref = O.delta_rule_grads(variant, f(inp["q"]), f(inp["k"]), f(inp["v"]), inp["g"], inp["beta"], inp["h0"], f(do), None,
                             use_qk_l2norm=l2)
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):
        if ref[name] is None:
            continue
        # same checkpoints, same adjoint (dbeta and dg are summed with atomics: equal up to summation order)
        if name in ("dbeta", "dg"):
            assert _rel(got[name], again[name]) <= 1e-5, name
        else:
            assert torch.equal(got[name], again[name]), name
        assert _rel(got[name], ref[name]) <= tol, (variant, name, _rel(got[name], ref[name]))


def test_autograd_uses_the_saved_states():
    from linearnexus_b200 import _lib
    inp = O.make_inputs("gated", 1, 2, 128, 128, 128, seed=4, io_dtype=torch.bfloat16)
    leaf = {k_: (None if v_ is None else v_.cuda().requires_grad_(v_.is_floating_point())) for k_, v_ in inp.items()}
    nf = _lib.launch_count()
    o, hT = L.gated_delta_rule_chunkwise(leaf["q"], leaf["k"], leaf["v"], leaf["g"], leaf["beta"])
    assert _lib.last_path() == "fwd_saving"
    # the forward that keeps the per-chunk states, with the adjoint's chunk-parallel pre-pass beside it
    assert _lib.launch_count() - nf == 2
    n0 = _lib.launch_count()
    (o.float().square().sum() + hT.sum()).backward()
    torch.cuda.synchronize()
    # adjoint + finalize only: no forward recomputation, no pre-pass (the path name is per host thread; autograd
    # runs elsewhere, so the launch counter is the witness)
    assert _lib.launch_count() - n0 == 2
    assert leaf["q"].grad is not None and torch.isfinite(leaf["q"].grad.float()).all()


@pytest.mark.parametrize("variant", ["gated", "delta"])
@pytest.mark.parametrize("K,V,T,Hq,H", [(16, 8, 70, 2, 2), (32, 40, 130, 1, 3), (48, 64, 64, 2, 4), (80, 24, 100, 1, 2),
                                        (96, 96, 65, 3, 3), (112, 16, 129, 1, 1), (128, 72, 257, 2, 4), (128, 128, 1, 1, 2)])
def test_tensor_core_backward_odd_shapes(variant, K, V, T, Hq, H):
    """bf16 inputs (tf32 tensor-core adjoint, 16 warps) against the exact fp32 path on the same values: channel
    counts that leave warps idle, value slices with a ragged last slice, ragged chunks, grouped q/k heads."""
    from linearnexus_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(K * 1000 + V)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    B = 2
    q, k, v = r(B, Hq, T, K).bfloat16(), r(B, Hq, T, K).bfloat16(), r(B, H, T, V).bfloat16()
    beta = torch.sigmoid(r(B, H, T))
    g = torch.nn.functional.logsigmoid(r(B, H, T) + 3) if variant == "gated" else None
    d_o, d_hT, h0 = (r(B, H, T, V) * 0.1).bfloat16(), r(B, H, K, V) * 0.1, r(B, H, K, V) * 0.05
    a = ops.chunk_backward(variant, q, k, v, g, beta, d_o, h0, d_hT)
    b = ops.chunk_backward(variant, q.float(), k.float(), v.float(), g, beta, d_o.float(), h0, d_hT)
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):
        if a[name] is None:
            continue
        x, y = a[name].float(), b[name].float()
        assert torch.isfinite(x).all(), name
        err = (x - y).abs().max() / y.abs().max().clamp_min(1e-20)
        assert err <= 2e-2, (name, float(err))   # the bf16 bar: max|x - ref| / max|ref|


def test_forward_of_grad_inputs_runs_for_shapes_the_backward_does_not_cover():
    """chunk_size 128 has a forward (token-recurrent kernel) but no backward: a call on requires_grad inputs still
    returns the forward result, and only .backward() reports the limit."""
    inp = O.make_inputs("gated", 1, 2, 256, 64, 64, seed=4)
    cu = {k: (None if v is None else v.cuda()) for k, v in inp.items()}
    q = cu["q"].clone().requires_grad_(True)
    o, hT = L.gated_delta_rule_chunkwise(q, cu["k"], cu["v"], cu["g"], cu["beta"], chunk_size=128)
    with torch.no_grad():
        o2, hT2 = L.gated_delta_rule_chunkwise(cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], chunk_size=128)
    assert torch.equal(o, o2) and torch.equal(hT, hT2)
    with pytest.raises(NotImplementedError, match="chunk_size <= 64"):
        o.sum().backward()


@pytest.mark.parametrize("variant", ["delta", "gated", "kda"])
@pytest.mark.parametrize("T", [17, 64, 65, 150, 320])
def test_gradients_without_the_initial_states(variant, T):
    """A training step without an initial state does not ask for its gradient: every other gradient stays the same, bit for bit."""
    inp = O.make_inputs(variant, 1, 3, T, 128, 128, seed=T, io_dtype=torch.bfloat16)
    cu = {k: None if t is None else t.cuda() for k, t in inp.items()}
    args = (variant, cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"])
    d_o = torch.randn(1, 3, T, 128, generator=torch.Generator().manual_seed(T)).cuda()
    d_hT = torch.randn(1, 3, 128, 128, generator=torch.Generator().manual_seed(T + 1)).cuda()
    for last in (None, d_hT):
        whole = ops.chunk_backward(*args, d_o, None, last, saved=ops.chunk_forward_saving(*args)[2])
        part = ops.chunk_backward(*args, d_o, None, last, saved=ops.chunk_forward_saving(*args)[2], _want_dh0=False)
        assert part.pop("dh0") is None and whole.pop("dh0") is not None
        for name, x in whole.items():
            assert x is part[name] is None or torch.equal(x, part[name]), name
    leaves = [None if t is None else t.clone().requires_grad_() for t in args[1:]]
    h0 = torch.zeros(1, 3, 128, 128, device="cuda")   # given, but no gradient wanted
    f = {"delta": lambda: L.delta_rule_chunkwise(leaves[0], leaves[1], leaves[2], leaves[4], h0),
         "gated": lambda: L.gated_delta_rule_chunkwise(*leaves, initial_state=h0), "kda": lambda: L.kda_chunkwise(*leaves, initial_state=h0)}[variant]
    f()[0].sum().backward()
    assert h0.grad is None and all(t is None or torch.isfinite(t.grad).all() for t in leaves)


@pytest.mark.parametrize("variant,B,Hq,H,T,bthd,strong", [
    ("gated", 1, 1, 1, 1, False, False), ("delta", 1, 2, 2, 63, True, False), ("gated", 1, 1, 2, 64, False, True),
    ("gated", 2, 1, 3, 65, True, False), ("delta", 1, 1, 2, 129, False, False), ("gated", 1, 2, 2, 200, True, True),
    ("gated", 3, 2, 2, 1665, False, False)])   # the last: 162 chunks, more than one per CTA
def test_local_pass_on_tcgen05(variant, B, Hq, H, T, bthd, strong):
    """Ragged chunks, one token, grouped q/k heads, both storages, a second chunk per persistent CTA, decays of e^-30 a token, against
    float64.  bf16 outputs round at 2^-9 (2-norm 1.7e-3); operands of the forward's checkpoints are bf16 too, in all 1e-2 of the largest."""
    inp = O.make_inputs(variant, B, H, T, 128, 128, seed=T, io_dtype=torch.bfloat16, h0_std=0.02)
    if variant == "delta":
        inp["k"] = torch.nn.functional.normalize(inp["k"].float(), dim=-1).bfloat16()
    if strong:
        inp["g"][:, :, ::5] = -30.0
    q, k = inp["q"][:, :Hq], inp["k"][:, :Hq]
    gen = torch.Generator().manual_seed(T + 1)
    do, dhT = torch.randn(B, H, T, 128, generator=gen).bfloat16(), torch.randn(B, H, 128, 128, generator=gen) * 0.1
    def cu(x):
        if x is None:
            return None
        return x.transpose(1, 2).contiguous().cuda().transpose(1, 2) if bthd else x.contiguous().cuda()
    l2 = variant != "delta"
    args = (variant, cu(q), cu(k), cu(inp["v"]), cu(inp["g"]), cu(inp["beta"]), cu(do))
    run = lambda: ops.chunk_backward(*args, initial_state=inp["h0"].cuda(), d_final_state=dhT.cuda(), chunk_size=64, use_qk_l2norm=l2)
    got, again = run(), run()
    L.check_device_status()
    rep = lambda x: x.double().repeat_interleave(H // Hq, 1)
    d = lambda x: None if x is None else x.double()
    ref = O.delta_rule_grads(variant, rep(q), rep(k), d(inp["v"]), d(inp["g"]), d(inp["beta"]), d(inp["h0"]), d(do), d(dhT),
                             use_qk_l2norm=l2)
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):
        want = ref[name]
        if want is None:
            assert got[name] is None
            continue
        if name in ("dq", "dk"):
            want = want.view(B, Hq, H // Hq, T, 128).sum(2)
        assert torch.equal(got[name], again[name]), name
        err = (got[name].double().cpu() - want).norm() / want.norm()
        assert err <= 1e-2, (name, err)


@pytest.mark.parametrize("B,Hq,H,T,bthd,l2,decay", [
    (1, 1, 1, 1, False, True, None), (2, 1, 3, 65, True, True, None), (1, 2, 2, 130, False, False, -0.5), (1, 1, 2, 640, True, True, 30.0),
    (81, 1, 1, 1, False, True, None), (41, 1, 1, 65, True, True, 11.0), (1, 1, 2, 641, False, False, None), (1, 2, 2, 703, False, True, 11.0),
    (1, 2, 2, 704, True, True, 11.2), (1, 1, 2, 800, True, True, 30.0), (1, 2, 2, 730, False, False, -0.5),
    (3, 2, 2, 1665, False, True, 40.0)])   # the last: 162 chunks, more than one per CTA
def test_kda_local_passes(B, Hq, H, T, bthd, l2, decay):
    """KDA: chunks that decay by at most 2^16 (11.09 nats) in every channel take the tcgen05 kernels, the others -- those with a positive
    log decay, and all of at most 80 in sequences of at most ten -- the ones with 16-row blocks; ragged chunks, grouped q/k heads, both storages, rows that are not normalised.  Against float64;
    bf16 outputs round at 2^-9 (2-norm 1.7e-3), operands of the forward's checkpoints are bf16 too, in all 1e-2 of the largest."""
    inp = O.make_inputs("kda", B, H, T, 128, 128, seed=T, io_dtype=torch.bfloat16, h0_std=0.02)
    if not l2:
        inp["k"] = (1.5 * torch.nn.functional.normalize(inp["k"].float(), dim=-1)).bfloat16()
        inp["beta"] = inp["beta"] * 0.5
    if decay is not None:   # one channel of the second chunk (of every other chunk of the long one)
        for t0 in range(64, T, 128):
            inp["g"][:, -1, t0:t0 + 64, 17] = -decay / 64
    q, k = inp["q"][:, :Hq], inp["k"][:, :Hq]
    gen = torch.Generator().manual_seed(T + 1)
    do, dhT = torch.randn(B, H, T, 128, generator=gen).bfloat16(), torch.randn(B, H, 128, 128, generator=gen) * 0.1
    def cu(x):
        return x.transpose(1, 2).contiguous().cuda().transpose(1, 2) if bthd else x.contiguous().cuda()
    args = ("kda", cu(q), cu(k), cu(inp["v"]), cu(inp["g"]), cu(inp["beta"]), cu(do))
    run = lambda: ops.chunk_backward(*args, initial_state=inp["h0"].cuda(), d_final_state=dhT.cuda(), chunk_size=64, use_qk_l2norm=l2)
    got, again = run(), run()
    L.check_device_status()
    rep = lambda x: x.double().repeat_interleave(H // Hq, 1)
    ref = O.delta_rule_grads("kda", rep(q), rep(k), inp["v"].double(), inp["g"].double(), inp["beta"].double(), inp["h0"].double(), do.double(),
                             dhT.double(), use_qk_l2norm=l2)
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):
        want = ref[name].view(B, Hq, H // Hq, T, 128).sum(2) if name in ("dq", "dk") else ref[name]
        assert torch.equal(got[name], again[name]), name
        err = (got[name].double().cpu() - want).norm() / want.norm()
        assert err <= 1e-2, (name, err)


@pytest.mark.parametrize("T,nats,loss", [(192, 0.4, "state"), (704, 0.25, "state"), (704, 0.4, "state"), (704, 1.0, "state"), (192, 0.6, "last"), (704, 0.25, "last"),
                                         (704, 0.6, "last")])
def test_kda_gradients_behind_chunks_that_decay_strongly(T, nats, loss):
    """Every channel of every token decays by `nats`; the loss is of the final state or of the last token alone, so what reaches the chunks before
    passes through N and Y of whole chunks, which are as small as the decay.  Chunk by chunk relative to itself, against float64: bf16 outputs
    round at 2^-9 (2-norm 1.7e-3), the others carry the error of the chunk's inverse (tf32 products: measured 1.2e-4 at most); four times that."""
    inp = O.make_inputs("kda", 1, 2, T, 128, 128, seed=T, io_dtype=torch.bfloat16, h0_std=0.02)
    inp["g"][...] = -nats
    gen = torch.Generator().manual_seed(1)
    do, dhT = torch.randn(1, 2, T, 128, generator=gen).bfloat16(), torch.randn(1, 2, 128, 128, generator=gen) * 0.1
    do[:, :, :T if loss == "state" else T - 1] = 0
    dhT = dhT if loss == "state" else None
    args = [inp[x] for x in ("q", "k", "v", "g", "beta")]
    got = ops.chunk_backward("kda", *(x.cuda() for x in args), do.cuda(), initial_state=inp["h0"].cuda(), d_final_state=None if dhT is None else dhT.cuda(),
                             chunk_size=64)
    L.check_device_status()
    ref = O.delta_rule_grads("kda", *(x.double() for x in args), inp["h0"].double(), do.double(), None if dhT is None else dhT.double())
    for name, tol in (("dq", 7e-3), ("dk", 7e-3), ("dv", 7e-3), ("dbeta", 5e-4), ("dg", 5e-4)):
        for t0 in range(0, T, 64):
            x, want = got[name][:, :, t0:t0 + 64].double().cpu(), ref[name][:, :, t0:t0 + 64]
            if want.norm() > 1e-33:   # (what is left of float32's and bf16's range)
                assert (x - want).norm() <= tol * want.norm(), (name, t0)
    if ref["dh0"].norm() > 1e-33:
        assert (got["dh0"].double().cpu() - ref["dh0"]).norm() <= 5e-4 * ref["dh0"].norm()


def _kda_backward(inp, do, dhT):
    """Gradients, and float64's (on the device: many sequences)."""
    cu = {n: x.cuda() for n, x in inp.items() if x is not None}
    args = [cu[n] for n in ("q", "k", "v", "g", "beta")]
    got = ops.chunk_backward("kda", *args, do.cuda(), initial_state=cu["h0"], d_final_state=dhT.cuda(), chunk_size=64)
    L.check_device_status()
    return got, O.delta_rule_grads("kda", *(x.double() for x in args), cu["h0"].double(), do.cuda().double(), dhT.cuda().double())


@pytest.mark.parametrize("T,beta,nats,tol", [(64, 1.0, None, 2e-4), (63, 1.0, 0.2, 2e-4), (64, 0.05, None, 3e-5), (64, 1.0, 0.43, 2e-4), (17, 1.0, None, 2e-4)])
def test_kda_float32_gradients_of_one_chunk(T, beta, nats, tol):
    """One chunk, its states in float32: no bf16 checkpoint between.  Operands are two bf16 terms, 2^-17 of every entry; at most four products follow
    each other (X, T, R or dVn, the gradient): 3e-5 where T is near I; its merges round to tf32, 2^-12 of its entries off the diagonal, of which those that
    add up to a gradient are most of it at most: 2e-4.  A term that is left out is 2^-9.  bf16 outputs round at 2^-9 (2-norm 1.7e-3)."""
    inp = O.make_inputs("kda", 81, 1, T, 128, 128, seed=T, io_dtype=torch.bfloat16, h0_std=0.02)
    inp["beta"] *= beta
    if nats is not None:
        inp["g"][...] = -nats
    gen = torch.Generator().manual_seed(T + 1)
    got, ref = _kda_backward(inp, torch.randn(81, 1, T, 128, generator=gen).bfloat16(), torch.randn(81, 1, 128, 128, generator=gen) * 0.1)
    for name, tol in (("dbeta", tol), ("dg", tol), ("dh0", tol), ("dq", 3e-3), ("dk", 3e-3), ("dv", 3e-3)):
        err = ((got[name].double() - ref[name]).norm() / ref[name].norm()).item()
        assert err <= tol, (name, err)


def test_kda_gradients_of_uneven_inputs():
    """Half of the value channels 2^-60 of the others, and one of another head infinite in one token: a value channel's gradients know nothing of the
    others, so each half keeps its own bits.  dv rounds to bf16; dh0 follows from N and Y, which T's tf32 merges decide: 2e-4."""
    T = 705
    inp = O.make_inputs("kda", 1, 2, T, 128, 128, seed=5, io_dtype=torch.bfloat16, h0_std=0.02)
    gen = torch.Generator().manual_seed(6)
    do, dhT = torch.randn(1, 2, T, 128, generator=gen).bfloat16(), torch.randn(1, 2, 128, 128, generator=gen) * 0.1
    for x in (inp["v"], inp["h0"], do, dhT):
        x[:, 0, :, 64:] *= 2.0 ** -60
    do[:, 1, 300, 5] = float("inf")
    got, ref = _kda_backward(inp, do, dhT)
    rest = [v for v in range(128) if v != 5]
    for name, tol in (("dv", 3e-3), ("dh0", 2e-4)):
        for x, want in ((got[name][:, 0, :, :64], ref[name][:, 0, :, :64]), (got[name][:, 0, :, 64:], ref[name][:, 0, :, 64:]),
                        (got[name][:, 1][..., rest], ref[name][:, 1][..., rest])):
            err = ((x.double() - want).norm() / want.norm()).item()
            assert err <= tol, (name, err)


@pytest.mark.parametrize("decay", [27.7, 27.75, 39.0])
def test_kda_local_passes_at_the_line(decay):
    """The line between the two kinds of chunks: 2^40 (27.726 nats) in any channel."""
    test_kda_local_passes(1, 2, 2, 703, True, True, decay)


def test_kda_wide_chunks_are_taken_one_by_one():
    """160 chunks past the line, two of 162 are not: every CTA of the kernels with 16-row blocks takes several of the list."""
    T = 1665
    inp = O.make_inputs("kda", 3, 2, T, 128, 128, seed=8, io_dtype=torch.bfloat16, h0_std=0.02)
    inp["g"] *= 20.0
    inp["g"][0, 0, 64:192] = -0.01
    gen = torch.Generator().manual_seed(9)
    got, ref = _kda_backward(inp, torch.randn(3, 2, T, 128, generator=gen).bfloat16(), torch.randn(3, 2, 128, 128, generator=gen) * 0.1)
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):   # bf16 operands in the forward's checkpoints: 1e-2 of the largest
        err = ((got[name].double() - ref[name]).norm() / ref[name].norm()).item()
        assert err <= 1e-2, (name, err)


@pytest.mark.parametrize("T,H", [(130, 2), (640, 8), (641, 2), (705, 27)])
def test_kda_decays_at_eight_bytes(T, H):
    """bf16 log decays whose rows start at eight bytes, where a tensor map does not take them: on both sides of the line of few chunks (ten a sequence, 80 in
    all) as with aligned ones, and from a forward that had them aligned.  Against float64: the bf16 budget of the other tests."""
    inp = O.make_inputs("kda", 1, H, T, 128, 128, seed=T, io_dtype=torch.bfloat16, h0_std=0.02, g_dtype=torch.bfloat16)
    gen = torch.Generator().manual_seed(T)
    do, dhT = torch.randn(1, H, T, 128, generator=gen).bfloat16().cuda(), (torch.randn(1, H, 128, 128, generator=gen) * 0.1).cuda()
    cu = {n: x.cuda() for n, x in inp.items()}
    apart = torch.empty(cu["g"].numel() + 4, dtype=torch.bfloat16, device="cuda")[4:].view_as(cu["g"]).copy_(cu["g"])
    assert apart.data_ptr() % 16 == 8 and apart.is_contiguous()
    def run(g, saved=None):
        r = ops.chunk_backward("kda", cu["q"], cu["k"], cu["v"], g, cu["beta"], do, initial_state=cu["h0"], d_final_state=dhT, chunk_size=64, saved=saved)
        L.check_device_status()
        return r
    ref = O.delta_rule_grads("kda", *(cu[n].double() for n in ("q", "k", "v", "g", "beta")), cu["h0"].double(), do.double(), dhT.double())
    want, got = run(cu["g"]), run(apart)
    save = lambda: ops.chunk_forward_saving("kda", cu["q"], cu["k"], cu["v"], cu["g"], cu["beta"], cu["h0"], chunk_size=64)[2]
    kept, again = run(cu["g"], save()), run(apart, save())
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):
        for x in (want, got, kept, again):
            assert (x[name].double() - ref[name]).norm() <= 1e-2 * ref[name].norm(), name
        assert torch.equal(kept[name], again[name]), name


def test_kda_two_backwards_behind_one_forward():
    """The saved workspace serves a second adjoint, chunks past the line included (they are taken from a list, which begins anew)."""
    T = 705
    inp = O.make_inputs("kda", 1, 2, T, 128, 128, seed=12, io_dtype=torch.bfloat16, h0_std=0.02)
    inp["g"][:, 1] *= 20.0
    cu = {n: x.cuda() for n, x in inp.items()}
    gen = torch.Generator().manual_seed(13)
    do, dhT = torch.randn(1, 2, T, 128, generator=gen).bfloat16().cuda(), (torch.randn(1, 2, 128, 128, generator=gen) * 0.1).cuda()
    args = [cu[n] for n in ("q", "k", "v", "g", "beta")]
    saved = ops.chunk_forward_saving("kda", *args, cu["h0"], chunk_size=64)[2]
    first, second = (ops.chunk_backward("kda", *args, do, initial_state=cu["h0"], d_final_state=dhT, chunk_size=64, saved=saved) for _ in range(2))
    L.check_device_status()
    ref = O.delta_rule_grads("kda", *(x.double() for x in args), cu["h0"].double(), do.double(), dhT.double())
    for name in ("dq", "dk", "dv", "dbeta", "dg", "dh0"):
        assert torch.equal(first[name], second[name]), name
        assert (first[name].double() - ref[name]).norm() <= 1e-2 * ref[name].norm(), name
