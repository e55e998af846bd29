"""The work this package is used for, as cases that can be timed and compared.

Four kinds, all through the public entry points:

``train``    ``flash_cuda.flash_attn`` forward and backward, as the attention mixer calls it in a training step:
             every mask (causal, sliding window with sinks, block-causal), head dim and dtype it takes.
``forward``  the same without gradients: evaluation and prefill.
``layer``    one mixer layer around its projections, forward and backward under autocast: QK-norm + RoPE of q and of
             k, value-residual blend, attention core, head gate.
``cached``   ``flash_cuda.flash_attn_cached``: an active block over [cache | block], the samplers' decode step.

Tensors are N(0, 1), what normalised queries and keys are and what the benchmark configurations prescribe.
"""
from __future__ import annotations

import math

import torch

from machinelearning_b200 import flash_cuda, qk_prologue, value_gate

DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}

# The most one drawn case may cost, next to the largest listed ones: arithmetic on the tensor cores, arithmetic
# in fp32 (which runs at a small fraction of that rate), and elements of q.
MOST_FLOPS = {"bf16": 3.0e13, "fp16": 3.0e13, "fp32": 1.0e11}
MOST_ELEMENTS = 1 << 27


def _case(name, kind, dtype, B, T, H, Hkv, D, window=0, sinks=0, block=0, keys=0, causal=True):
    c = {"kind": kind, "dtype": dtype, "B": B, "T": T, "H": H, "Hkv": Hkv, "D": D, "window": window, "sinks": sinks,
         "block": block, "keys": keys, "causal": causal}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a unit-test sized model: a call is a few microseconds of work, so what counts is getting it launched
        _case("train_tiny", "train", "bf16", 2, 100, 4, 2, 64),
        # the fp32 configuration: training without autocast
        _case("train_fp32", "train", "fp32", 4, 256, 4, 4, 64),
        # the self-check's default shape (grouped heads of 32), in half precision
        _case("train_gqa_d32", "train", "fp16", 8, 1024, 12, 4, 32),
        # diffusion / semi-autoregressive training: block-causal mask, a length that is no multiple of a tile
        _case("train_block_causal", "train", "fp16", 6, 1000, 12, 4, 64, block=32),
        # the 124M model's layer in bf16: the benchmark's default workload
        _case("train_causal", "train", "bf16", 32, 1024, 12, 12, 64),
        # heads of 128 at a medium length, grouped
        _case("train_d128", "train", "bf16", 4, 2048, 12, 4, 128),
        # the sliding-window mixer
        _case("train_window", "train", "bf16", 16, 4096, 16, 16, 64, window=256),
        # long-context training, the largest call
        _case("train_long", "train", "bf16", 8, 16384, 16, 16, 128),
        # prefill / evaluation of one long prompt of odd length
        _case("prefill", "forward", "bf16", 1, 8191, 16, 4, 128),
        # one layer of the 124M model at a per-GPU batch of 16: the elementwise steps around the core count as much
        _case("layer", "layer", "bf16", 16, 1024, 12, 12, 64),
        # decoding one sequence in blocks of 32 tokens: latency
        _case("decode_one", "cached", "bf16", 1, 32, 12, 12, 64, keys=1056),
        # decoding against a long cache: the cache's bandwidth
        _case("decode_long", "cached", "bf16", 1, 64, 16, 16, 128, keys=16448),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["train"] * 5 + ["forward"] * 2 + ["layer"] * 2 + ["cached"] * 3)
    dtype = rng.choice(["bf16"] * 4 + ["fp16"] * 2 + ["fp32"])
    D = rng.choice([32, 64, 64, 128])
    Hkv = rng.choice([1, 2, 4, 8, 12, 16])
    H = Hkv * rng.choice([g for g in (1, 1, 2, 3, 4) if Hkv * g <= 16])
    if kind == "cached":
        # blocks of 1 to 128 tokens over up to 16k cached keys; a window's cache holds little more than the window
        T, keys = _log_int(rng, 1, 128), _log_int(rng, 64, 16384)
        B = _log_int(rng, 1, max(1, min(16, (MOST_ELEMENTS >> 1) // (keys * Hkv * D))))
        window, sinks, causal = 0, 0, rng.random() < 0.7
        if rng.random() < 0.3:
            window, causal = _log_int(rng, 32, 2048), True
            sinks = rng.choice([0, 4]) if window > 4 else 0
            keys = min(keys, window)
        return _case("", kind, dtype, B, T, H, Hkv, D, window, sinks, 0, keys + T, causal)
    T = _log_int(rng, 32, 4096 if dtype == "fp32" or kind == "layer" else 16384)
    window = sinks = block = 0
    mask = rng.choice(["causal"] * 3 + ["window", "block"])
    if mask == "window":
        window = _log_int(rng, 16, 2048)
        sinks = rng.choice([0, 0, 4]) if window > 4 else 0
    elif mask == "block":
        block = _log_int(rng, 8, 1024)
    one = _case("", kind, dtype, 1, T, H, Hkv, D, window, sinks, block)
    most = min(MOST_ELEMENTS // (T * H * D), int(MOST_FLOPS[dtype] / work(one)["flops"]), 64)
    one["B"] = _log_int(rng, 1, max(1, most))
    return one


def _pairs(c):
    """Visible (query, key) pairs of one head."""
    T, w, b = c["T"], c["window"], c["block"]
    if c["kind"] == "cached":
        old = c["keys"] - T
        if w:
            return sum(min(w, old + t + 1) for t in range(T))
        return sum(old + t + 1 for t in range(T)) if c["causal"] else T * c["keys"]
    if w and w < T:
        return w * (w + 1) // 2 + (T - w) * w
    if b:
        return sum(min(b, T - q) * min(T, q + b) for q in range(0, T, b))
    return T * (T + 1) // 2


def work(case):
    c = case
    size = 4 if c["dtype"] == "fp32" else 2
    B, T, H, Hkv, D = c["B"], c["T"], c["H"], c["Hkv"], c["D"]
    nq, nkv, rows = B * T * H * D, B * T * Hkv * D, B * T * H
    products = 4 * D * _pairs(c) * B * H                          # S = Q K^T and O = P V
    if c["kind"] == "cached":
        return {"bytes": size * (2 * nq + 2 * B * Hkv * c["keys"] * D), "flops": products}
    if c["kind"] == "forward":
        return {"bytes": size * (2 * nq + 2 * nkv), "flops": products}
    if c["kind"] == "train":                                      # q, k, v, dO in; O, dQ, dK, dV out
        return {"bytes": size * (4 * nq + 4 * nkv), "flops": 14 * D * _pairs(c) * B * H}
    # layer: q, k, v, v0, the gate's logits and the upstream gradient in; the result and six gradients out
    return {"bytes": size * (4 * nq + 6 * nkv + 2 * rows), "flops": 14 * D * _pairs(c) * B * H + 30 * nq + 40 * nkv}


def tolerance(case):
    return {"rel": 1e-5 if case["dtype"] == "fp32" else 1e-2}


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype = DTYPES[c["dtype"]]
    B, T, H, Hkv, D = c["B"], c["T"], c["H"], c["Hkv"], c["D"]
    randn = lambda *shape: torch.randn(*shape, device="cuda", dtype=torch.float32, generator=g)  # noqa: E731
    s = {"case": c, "scale": 1.0 / math.sqrt(D)}
    if c["kind"] == "cached":
        L = c["keys"]
        s["q"] = randn(B, T, H, D).to(dtype)
        s["k"], s["v"] = randn(B, Hkv, L, D).to(dtype), randn(B, Hkv, L, D).to(dtype)
        s["qpos"] = s["kpos"] = None
        if c["window"]:
            # a sampler that evicts hands over absolute positions: the sinks, then the tail the window reaches
            first = 3 * L
            held = L - T
            kept = min(c["sinks"], held)
            old = torch.cat([torch.arange(kept), torch.arange(first - (held - kept), first)])
            s["qpos"] = torch.arange(first, first + T).cuda()
            s["kpos"] = torch.cat([old, torch.arange(first, first + T)]).cuda()
        return s
    grad = c["kind"] != "forward"
    s["q"] = randn(B, T, H, D).to(dtype).requires_grad_(grad)
    s["k"] = randn(B, T, Hkv, D).to(dtype).requires_grad_(grad)
    s["v"] = randn(B, T, Hkv, D).to(dtype).requires_grad_(grad)
    if not grad:
        return s
    up = randn(B, T, H, D)
    if c["kind"] == "layer":
        s["v0"] = randn(B, T, Hkv, D).to(dtype).requires_grad_()
        s["q_weight"] = (1 + 0.1 * randn(D)).requires_grad_()
        s["k_weight"] = (1 + 0.1 * randn(D)).requires_grad_()
        s["lam"] = (0.5 * randn(1)).requires_grad_()
        s["gate"] = randn(B, T, H).to(dtype).requires_grad_()
        half = torch.arange(0, D, 2, device="cuda").float() / D
        angle = torch.outer(torch.arange(T, device="cuda").float(), 10000.0 ** -half)
        angle = torch.cat((angle, angle), dim=-1)
        s["cos"], s["sin"] = angle.cos(), angle.sin()
        # a loss gradient points along what the blend mixes, so the blend's own gradient is no sum of pure noise
        up = up + 0.25 * (s["v0"] - s["v"]).detach().float().repeat_interleave(H // Hkv, dim=2)
    s["up"] = up.to(dtype)
    return s


def _attention(s, q, k, v):
    c = s["case"]
    return flash_cuda.flash_attn(q, k, v, s["scale"], window=c["window"], sinks=c["sinks"], block=c["block"])


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "cached":
        with torch.no_grad():
            return flash_cuda.flash_attn_cached(s["q"], s["k"], s["v"], s["scale"], qpos=s["qpos"], kpos=s["kpos"],
                                                causal=c["causal"], window=c["window"], sinks=c["sinks"])
    if c["kind"] == "forward":
        with torch.no_grad():
            return _attention(s, s["q"], s["k"], s["v"])
    if c["kind"] == "train":
        y = _attention(s, s["q"], s["k"], s["v"])
        return (y.detach(), *torch.autograd.grad(y, (s["q"], s["k"], s["v"]), s["up"]))
    with torch.autocast("cuda", dtype=DTYPES[c["dtype"]], enabled=c["dtype"] != "fp32"):
        q = qk_prologue.qk_prologue(s["q"], s["q_weight"], s["cos"], s["sin"])
        k = qk_prologue.qk_prologue(s["k"], s["k_weight"], s["cos"], s["sin"])
        v = value_gate.value_blend(s["v"], s["v0"], s["lam"])
        y = value_gate.head_gate(_attention(s, q, k, v), s["gate"])
    leaves = tuple(s[n] for n in ("q", "k", "v", "v0", "q_weight", "k_weight", "lam", "gate"))
    return (y.detach(), *torch.autograd.grad(y, leaves, s["up"]))
