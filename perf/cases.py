"""The work this package is measured on: public calls over the sizes, types and options they are used with.

A case names a ``kind`` and its sizes.  The kinds:

* ``decode``   one token per sequence, the float32 state cache updated in place (serving, one layer).
* ``block``    what one Gated DeltaNet layer runs between its projections: short convolutions with SiLU, gate
               activations, the delta-rule op, gated RMS norm -- over a prompt, or over one token with caches.
* ``prefill``  the chunkwise op alone, every variant, bf16 or float32.
* ``packed``   the chunkwise op over a packed batch of prompts of different lengths.
* ``train``    forward and backward of the chunkwise op through autograd.
* ``scan``     the RWKV-7, RWKV-6 and Mamba-2 state scans.

Values follow the distributions of the repository's benchmark: q, k normal and l2-normalised, v normal,
beta = sigmoid(normal), log decay = logsigmoid(normal + 4); states normal with deviation 0.02.
"""
import math
import random

import torch
import torch.nn.functional as F

import linearnexus_b200 as L

D = 128          # head dimension of the bf16 models
CHUNK = 64
CONV = 4         # short-convolution window


def listed():
    return [
        # one user's chat, one layer: nothing but latency
        {"name": "decode_single", "kind": "decode", "variant": "gated", "B": 1, "H": 16, "Hq": 16},
        # a full serving batch: 537 MB of state read and written per step
        {"name": "decode_batch", "kind": "decode", "variant": "gated", "B": 256, "H": 32, "Hq": 32},
        # a whole layer's token step for a moderate batch, conv caches and state in place
        {"name": "block_step", "kind": "block", "B": 32, "T": 1, "H": 16, "Hq": 16},
        # a whole layer over one prompt of odd length, grouped q/k heads, token-major storage
        {"name": "block_prompt", "kind": "block", "B": 1, "T": 1777, "H": 16, "Hq": 8},
        # the benchmark's Gated DeltaNet forward
        {"name": "gated_prefill", "kind": "prefill", "variant": "gated", "dtype": "bf16", "layout": "bhtd", "h0": False,
         "B": 8, "T": 4096, "H": 16, "Hq": 16, "D": 128},
        # the benchmark's KDA forward, continued from a state
        {"name": "kda_prefill", "kind": "prefill", "variant": "kda", "dtype": "bf16", "layout": "bhtd", "h0": True,
         "B": 4, "T": 8192, "H": 32, "Hq": 32, "D": 128},
        # the benchmark's float32 DeltaNet forward
        {"name": "delta_fp32", "kind": "prefill", "variant": "delta", "dtype": "fp32", "layout": "bhtd", "h0": False,
         "B": 2, "T": 512, "H": 4, "Hq": 4, "D": 64},
        # prompts of different lengths in one batch (continuous batching)
        {"name": "packed_prompts", "kind": "packed", "variant": "gated", "seqs": 16, "total": 9000, "H": 16, "Hq": 16,
         "split": 1},
        # one GPU's share of the benchmark's training step
        {"name": "gated_train", "kind": "train", "variant": "gated", "layout": "bhtd", "B": 2, "T": 4096, "H": 16},
        # the same step with per-channel decay
        {"name": "kda_train", "kind": "train", "variant": "kda", "layout": "bhtd", "B": 2, "T": 4096, "H": 16},
        # the benchmark's RWKV-7 and Mamba-2 scans
        {"name": "rwkv7_scan", "kind": "scan", "rule": "rwkv7", "B": 8, "T": 4096, "H": 16, "K": 64, "V": 64, "groups": 1},
        {"name": "mamba2_scan", "kind": "scan", "rule": "mamba2", "B": 8, "T": 4096, "H": 16, "K": 128, "V": 64, "groups": 1},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "block", "block", "prefill", "prefill", "prefill", "packed", "train", "train", "scan", "scan"])
    if kind == "decode":
        H = rng.choice([4, 8, 16, 32])
        return {"kind": kind, "variant": rng.choice(["gated", "gated", "kda", "delta"]), "B": _log_int(rng, 1, 256), "H": H,
                "Hq": rng.choice([H, H // 2])}
    if kind == "block":
        H = rng.choice([4, 8, 16])
        Hq = rng.choice([H, H // 2])
        if rng.random() < 0.4:
            return {"kind": kind, "B": _log_int(rng, 1, 128), "T": 1, "H": H, "Hq": Hq}
        B = rng.choice([1, 1, 2, 4])
        return {"kind": kind, "B": B, "T": _log_int(rng, 65, 8192 // B), "H": H, "Hq": Hq}
    if kind == "prefill":
        variant = rng.choice(["gated", "gated", "kda", "delta"])
        layout = rng.choice(["bhtd", "bthd"])
        h0 = rng.random() < 0.5
        if rng.random() < 0.3:   # float32: evaluation and small models
            d, H = rng.choice([64, 64, 128]), rng.choice([2, 4, 8])
            B = rng.choice([1, 2, 4])
            return {"kind": kind, "variant": variant, "dtype": "fp32", "layout": layout, "h0": h0, "B": B,
                    "T": _log_int(rng, 32, 2048 // B), "H": H, "Hq": H, "D": d}
        H = rng.choice([4, 8, 16, 32])
        B = _log_int(rng, 1, 8)
        most = (4 * 8192 * 32 if variant == "kda" else 8 * 4096 * 16) // (B * H)
        return {"kind": kind, "variant": variant, "dtype": "bf16", "layout": layout, "h0": h0, "B": B,
                "T": _log_int(rng, 64, min(8192, most)), "H": H, "Hq": rng.choice([H, H, H // 2]), "D": D}
    if kind == "packed":
        seqs = rng.randint(4, 24)
        return {"kind": kind, "variant": rng.choice(["gated", "gated", "kda"]), "seqs": seqs,
                "total": _log_int(rng, 64 * seqs, 16384), "H": rng.choice([8, 16]), "Hq": 8, "split": rng.randrange(1 << 20)}
    if kind == "train":
        H = rng.choice([4, 8, 16])
        B = rng.choice([1, 2, 4])
        return {"kind": kind, "variant": rng.choice(["gated", "kda", "delta"]), "layout": rng.choice(["bhtd", "bthd"]), "B": B,
                "T": _log_int(rng, 256, min(4096, 8192 * 16 // (B * H))), "H": H}
    rule = rng.choice(["rwkv7", "rwkv6", "mamba2"])
    H = rng.choice([8, 16, 32])
    B = _log_int(rng, 1, 8)
    return {"kind": kind, "rule": rule, "B": B, "T": _log_int(rng, 64, min(4096, 8 * 4096 * 16 // (B * H))), "H": H,
            "K": rng.choice([64, 128]) if rule == "mamba2" else 64, "V": 64, "groups": rng.choice([1, 2]) if rule == "mamba2" else 1}


def _lengths(case):
    """Prompt lengths of a packed case: at least 16 tokens each, spread unevenly, adding up to `total`."""
    n, total = case["seqs"], case["total"]
    rng = random.Random(case["split"])
    w = [math.exp(rng.gauss(0.0, 0.8)) for _ in range(n)]
    spare = total - 16 * n
    lens = [16 + int(spare * x / sum(w)) for x in w]
    lens[0] += total - sum(lens)
    return lens


# ---- inputs -----------------------------------------------------------------------------------------------------------

class _Rand:
    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def __call__(self, *shape, dtype=torch.float32, scale=1.0):
        x = torch.randn(*shape, generator=self.gen, device="cuda")
        if scale != 1.0:
            x.mul_(scale)
        return x.to(dtype)

    def unit(self, *shape, dtype=torch.float32):
        return F.normalize(torch.randn(*shape, generator=self.gen, device="cuda"), dim=-1).to(dtype)

    def decay(self, *shape):
        return F.logsigmoid(torch.randn(*shape, generator=self.gen, device="cuda") + 4.0)

    def gate(self, *shape):
        return torch.sigmoid(torch.randn(*shape, generator=self.gen, device="cuda"))


def _qkvgb(r, variant, lead, Hq, H, K, V, dtype):
    """q, k, v, g, beta with the given leading shape (heads last before the feature axis)."""
    g = None if variant == "delta" else r.decay(*lead, H) if variant == "gated" else r.decay(*lead, H, K)
    return [r.unit(*lead, Hq, K, dtype=dtype), r.unit(*lead, Hq, K, dtype=dtype), r(*lead, H, V, dtype=dtype), g, r.gate(*lead, H)]


def _sequence_inputs(r, case, variant, H, Hq, K, dtype):
    """[B,H,T,...] inputs, contiguous or as views of token-major arrays."""
    B, T = case["B"], case["T"]
    xs = [None if x is None else x.transpose(1, 2) for x in _qkvgb(r, variant, (B, T), Hq, H, K, K, dtype)]
    return xs if case["layout"] == "bthd" else [None if x is None else x.contiguous() for x in xs]


def prepare(case, seed):
    r, kind = _Rand(seed), case["kind"]
    st = {"case": case}
    if kind == "decode":
        B, H = case["B"], case["H"]
        st["x"] = _qkvgb(r, case["variant"], (B,), case["Hq"], H, D, D, torch.bfloat16)
        st["S"] = r(B, H, D, D, scale=0.02)
    elif kind == "block":
        B, T, H, Hq = case["B"], case["T"], case["H"], case["Hq"]
        bf = torch.bfloat16
        st["qkv"] = [r(B, T, n * D, dtype=bf) for n in (Hq, Hq, H)]        # projections of the hidden states
        st["ab"] = [r(B, T, H, dtype=bf), r(B, T, H, dtype=bf)]
        st["gate"] = r(B, T, H, D, dtype=bf)
        st["conv"] = [r(CONV, n * D, scale=0.5) for n in (Hq, Hq, H)]       # parameters, float32
        st["A_log"], st["dt_bias"] = r(H, scale=0.5) - 1.0, r(H, scale=0.5) - 3.0
        st["norm"] = 1.0 + r(D, scale=0.1)
        if T == 1:
            st["cache"] = [r(B, CONV - 1, n * D, dtype=bf) for n in (Hq, Hq, H)]
            st["S"] = r(B, H, D, D, scale=0.02)
    elif kind == "prefill":
        dtype = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
        st["x"] = _sequence_inputs(r, case, case["variant"], case["H"], case["Hq"], case["D"], dtype)
        st["h0"] = r(case["B"], case["H"], case["D"], case["D"], scale=0.02) if case["h0"] else None
    elif kind == "packed":
        lens = _lengths(case)
        st["cu"] = [sum(lens[:i]) for i in range(len(lens) + 1)]
        st["x"] = _qkvgb(r, case["variant"], (case["total"],), case["Hq"], case["H"], D, D, torch.bfloat16)
    elif kind == "train":
        H = case["H"]
        st["x"] = [None if x is None else x.detach().requires_grad_(True)
                   for x in _sequence_inputs(r, case, case["variant"], H, H, D, torch.bfloat16)]
        d_o = r(case["B"], case["T"], H, D, dtype=torch.float32 if case["variant"] == "kda" else torch.bfloat16).transpose(1, 2)
        st["d_o"] = d_o if case["layout"] == "bthd" else d_o.contiguous()
    else:
        B, T, H, K, V, bf = case["B"], case["T"], case["H"], case["K"], case["V"], torch.bfloat16
        if case["rule"] == "rwkv7":
            kk = r.unit(B, H, T, K)
            st["x"] = [r(B, H, T, K, dtype=bf), r(B, H, T, K, dtype=bf, scale=0.5), r(B, H, T, V, dtype=bf), (-kk).to(bf),
                       (kk * r.gate(B, H, T, K)).to(bf), (-torch.exp(r(B, H, T, K) - 1.0)).to(bf)]
            st["h0"] = r(B, H, K, V, scale=0.02)
        elif case["rule"] == "rwkv6":
            st["x"] = [r(B, H, T, K, dtype=bf), r(B, H, T, K, dtype=bf, scale=0.5), r(B, H, T, V, dtype=bf),
                       (-r(B, H, T, K).abs() - 0.5).to(bf), r(H, K, scale=0.5)]
            st["h0"] = r(B, H, K, V, scale=0.02)
        else:
            G = case["groups"]
            st["x"] = [r(B, T, H, V, dtype=bf), r(B, T, H, scale=0.5), -torch.exp(r(H, scale=0.5)),
                       r(B, T, G, K, dtype=bf, scale=0.5), r(B, T, G, K, dtype=bf, scale=0.5), r(H)]
            st["dt_bias"] = r(H, scale=0.3)
            st["h0"] = r(B, H, V, K, scale=0.02)
    return st


# ---- one pass -----------------------------------------------------------------------------------------------------------

def _chunkwise(variant, q, k, v, g, beta, h0=None):
    if variant == "delta":
        return L.delta_rule_chunkwise(q, k, v, beta, h0, chunk_size=CHUNK)
    op = L.gated_delta_rule_chunkwise if variant == "gated" else L.kda_chunkwise
    return op(q, k, v, g, beta, initial_state=h0, chunk_size=CHUNK)


def _block(st):
    case = st["case"]
    B, T, H, Hq = case["B"], case["T"], case["H"], case["Hq"]
    step = T == 1
    qkv, caches = [], []
    for i, n in enumerate((Hq, Hq, H)):
        cache = st["cache"][i] if step else None
        y, c = L.short_conv_silu(st["qkv"][i], st["conv"][i], cache=cache, cache_out=cache)
        qkv.append(y.view(B, T, n, D))
        caches.append(c)
    g, beta = L.gated_deltanet_gates(st["ab"][0], st["ab"][1], st["A_log"], st["dt_bias"])
    if step:
        o, S = L.gated_delta_rule_step(*(x[:, 0] for x in qkv), g[:, 0], beta[:, 0], st["S"], inplace=True)
        o = o[:, :, None]
    else:
        q, k, v = (x.transpose(1, 2) for x in qkv)
        o, S = L.gated_delta_rule_chunkwise(q, k, v, g.transpose(1, 2), beta.transpose(1, 2), chunk_size=CHUNK)
    return L.rmsnorm_gated(o, st["norm"], st["gate"]), S, caches


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "block":
        return _block(st)
    if kind == "scan":
        x, h0 = st["x"], st["h0"]
        if case["rule"] == "rwkv7":
            return L.dplr_delta_rule_recurrent(*x, scale=case["K"] ** -0.5, initial_state=h0)
        if case["rule"] == "rwkv6":
            return L.rwkv6_recurrent(*x, scale=case["K"] ** -0.5, initial_state=h0)
        return L.ssd_chunk_scan(*x, chunk_size=256, n_groups=case["groups"], ssm_state=h0, dt_bias=st["dt_bias"],
                                dt_limit=(0.001, 5.0))
    q, k, v, g, beta = st["x"]
    variant = case["variant"]
    if kind == "decode":
        if variant == "delta":
            o, st["S"] = L.delta_rule_step(q, k, v, beta, st["S"])
            return o, st["S"]
        step = L.gated_delta_rule_step if variant == "gated" else L.kda_step
        return step(q, k, v, g, beta, st["S"], inplace=True)
    if kind == "prefill":
        return _chunkwise(variant, q, k, v, g, beta, st["h0"])
    if kind == "packed":
        return L.chunkwise_varlen(variant, q, k, v, g, beta, st["cu"])
    o, hT = _chunkwise(variant, q, k, v, g, beta)
    leaves = [x for x in st["x"] if x is not None]
    return [o.detach(), hT.detach(), *torch.autograd.grad(o, leaves, st["d_o"])]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

def _scan_work(tokens, units, Hq, H, K, V, variant, io, out, h0):
    """Bytes and flops of the chunk form over `tokens` tokens of H heads (`units` states): inputs and outputs once; the
    products of a chunk (6 C K + 4 C V + 6 K V + C^2 / 3 per token and head)."""
    g = 0 if variant == "delta" else 4 if variant == "gated" else 4 * K
    nbytes = tokens * (2 * Hq * K * io + H * (V * io + V * out + g + 4)) + units * 4 * K * V * (2 if h0 else 1)
    return nbytes, tokens * H * (6 * CHUNK * K + 4 * CHUNK * V + 6 * K * V + CHUNK * CHUNK / 3)


def work(case):
    kind, H = case["kind"], case["H"]
    if kind == "decode":
        units, g = case["B"] * H, {"delta": 0, "gated": 4, "kda": 4 * D}[case["variant"]]
        out = 4 if case["variant"] == "kda" else 2
        return {"bytes": units * (8 * D * D + 2 * D + out * D + g + 4) + case["B"] * case["Hq"] * 4 * D, "flops": units * 8 * D * D}
    if kind == "block":
        B, T, Hq = case["B"], case["T"], case["Hq"]
        C = (2 * Hq + H) * D
        tokens = B * T
        nbytes = tokens * (2 * C + 4 * H + 2 * H * D + 2 * H * D) + B * (CONV - 1) * 2 * C + 4 * CONV * C + B * H * 4 * D * D
        flops = tokens * (2 * CONV * C + 8 * H * D)
        if T == 1:
            return {"bytes": nbytes + B * (CONV - 1) * 2 * C + B * H * 4 * D * D, "flops": flops + B * H * 8 * D * D}
        return {"bytes": nbytes, "flops": flops + _scan_work(tokens, B * H, Hq, H, D, D, "gated", 2, 2, False)[1]}
    if kind == "prefill":
        io = 4 if case["dtype"] == "fp32" else 2
        b, f = _scan_work(case["B"] * case["T"], case["B"] * H, case["Hq"], H, case["D"], case["D"], case["variant"], io,
                          4 if case["variant"] == "kda" else io, case["h0"])
        return {"bytes": b, "flops": f}
    if kind == "packed":
        b, f = _scan_work(case["total"], case["seqs"] * H, case["Hq"], H, D, D, case["variant"], 2,
                          4 if case["variant"] == "kda" else 2, False)
        return {"bytes": b, "flops": f}
    if kind == "train":
        tokens, out = case["B"] * case["T"], 4 if case["variant"] == "kda" else 2
        g = {"delta": 0, "gated": 4, "kda": 4 * D}[case["variant"]]
        # inputs and the output gradient in; output, final state and the inputs' gradients out
        nbytes = tokens * H * (2 * (6 * D + g + 4) + 2 * out * D) + case["B"] * H * 4 * D * D
        return {"bytes": nbytes, "flops": 3 * _scan_work(tokens, 1, H, H, D, D, case["variant"], 2, out, False)[1]}
    B, T, K, V = case["B"], case["T"], case["K"], case["V"]
    state = B * H * 8 * K * V
    if case["rule"] == "mamba2":
        return {"bytes": B * T * (H * (4 * V + 4) + case["groups"] * 4 * K) + state, "flops": B * T * H * 5 * K * V}
    n, f = (5, 9) if case["rule"] == "rwkv7" else (3, 7)
    return {"bytes": B * H * T * 2 * (n * K + 2 * V) + state, "flops": B * H * T * f * K * V}


def tolerance(case):
    kind = case["kind"]
    if kind == "prefill" and case["dtype"] == "fp32":
        return {"rel": 1e-5}                       # float32 sums in another order
    if kind == "decode":
        return {"rel": 1e-5 if case["variant"] == "kda" else 4e-3}   # float32 arithmetic; bf16 outputs
    if kind == "scan":
        return {"rel": 4e-3}                       # float32 arithmetic, bf16 outputs
    return {"rel": 1e-2}                           # bf16 operands, float32 accumulation
