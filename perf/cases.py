"""The work this library is asked to do, as cases that a timing program can run one by one.

A case is a dict of plain values.  Three operations of the public namespace appear, each as a program calls it:

``attention``  ``scaled_dot_product_attention``: inference (forward only) and training (forward, then the gradients
               of q, k, v and, where the bias is learned, of the bias), fp32 / bf16 / fp16, head dims 32 to 128,
               bias per (batch, head), shared over the batch or per key, masks per key or per (query, key), causal,
               lengths on and off the 128-wide tiles, QK-norm
``layer_norm``      forward and all gradients
``selective_scan``  forward, and forward with all gradients

``listed`` holds the five benchmark workloads of this repository, the one workload the reference publishes a time for,
and one or two ordinary shapes of each remaining option; ``draw`` gives further cases of the same ranges.
"""
from __future__ import annotations

import math

import torch

from nitrix_b200.nn import layer_norm, scaled_dot_product_attention, selective_scan

_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_BYTES = {"f32": 4, "bf16": 2, "f16": 2}


def _attention(name, *, dtype, B, H, S, D, T=None, train, bias="none", bias_grad=False, mask="none", causal=False,
               qk_norm=False):
    case = dict(op="attention", dtype=dtype, B=B, H=H, S=S, T=S if T is None else T, D=D, train=train, bias=bias,
                bias_grad=bias_grad, mask=mask, causal=causal, qk_norm=qk_norm)
    return dict(name=name, **case) if name else case


def _layer_norm(name, *, dtype, rows, C, train):
    case = dict(op="layer_norm", dtype=dtype, rows=rows, C=C, train=train)
    return dict(name=name, **case) if name else case


def _scan(name, *, dtype, B, L, C, N, train):
    case = dict(op="selective_scan", dtype=dtype, B=B, L=L, C=C, N=N, train=train)
    return dict(name=name, **case) if name else case


def listed():
    return [
        # the smallest training step: a short fp32 window with a learned bias and padded keys; launches count
        _attention("f32_window_train", dtype="f32", B=2, H=4, S=256, D=64, train=True, bias="full", bias_grad=True,
                   mask="key"),
        # fp32 inference at the shape the reference publishes a wall time for
        _attention("f32_infer_s344", dtype="f32", B=4, H=6, S=344, D=64, train=False),
        # an fp32 training step that fills the GPU
        _attention("f32_train_s1024", dtype="f32", B=8, H=16, S=1024, D=64, train=True),
        # a language-model layer: causal, distance bias shared over the batch
        _attention("bf16_causal_shared_bias_train", dtype="bf16", B=8, H=16, S=2048, D=64, train=True, bias="shared",
                   causal=True),
        # a pair-biased layer: bias per (batch, head) with its gradient, dense boolean mask; the largest in bytes
        _attention("bf16_pair_bias_train", dtype="bf16", B=4, H=32, S=4096, D=128, train=True, bias="full",
                   bias_grad=True, mask="full"),
        # an encoder over a batch of sequences of unequal length
        _attention("f16_padded_train", dtype="f16", B=32, H=8, S=1024, D=64, train=True, mask="key"),
        # one very long causal sequence with a per-key bias; the largest in operations
        _attention("bf16_long_causal_train", dtype="bf16", B=1, H=16, S=65536, D=128, train=True, bias="key",
                   causal=True),
        # windowed vision attention: many short odd-length windows, relative-position bias learned over the batch
        _attention("bf16_windows_shared_bias_train", dtype="bf16", B=32, H=8, S=217, D=64, train=True, bias="shared",
                   bias_grad=True),
        # cross-attention inference with QK-norm, ragged on both sides, padded keys
        _attention("bf16_cross_qk_norm_infer", dtype="bf16", B=8, H=16, S=197, T=1111, D=128, train=False, mask="key",
                   qk_norm=True),
        # a wide transformer layer's norm, forward and backward
        _layer_norm("bf16_layer_norm_train", dtype="bf16", rows=8192, C=8192, train=True),
        # a Mamba block's scan at model width 1024, training and inference
        _scan("f32_scan_train", dtype="f32", B=8, L=1024, C=2048, N=16, train=True),
        _scan("bf16_scan_infer", dtype="bf16", B=8, L=2048, C=2048, N=16, train=False),
    ]


# ---- further cases of the same ranges ------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A length spread over the logarithm of the range; half of them multiples of 64, the rest as they fall."""
    n = _log_int(rng, lo, hi)
    if rng.random() < 0.5:
        n = min(hi, max(64, round(n / 64) * 64))
    return n


def draw(rng):
    op = rng.choice(["attention"] * 6 + ["layer_norm", "selective_scan"])
    if op == "layer_norm":
        dtype = rng.choice(["bf16", "f16", "f32"])
        C = _log_int(rng, 64, 8192)
        if rng.random() < 0.75:
            C = max(64, C // 64 * 64)
        rows = _log_int(rng, 256, 32768)
        return _layer_norm(None, dtype=dtype, rows=rows, C=C, train=rng.random() < 0.7)
    if op == "selective_scan":
        return _scan(None, dtype=rng.choice(["f32", "bf16", "f16"]), B=rng.randint(1, 8), L=_log_int(rng, 128, 2048),
                     C=_log_int(rng, 128, 2048), N=rng.choice([8, 16, 16, 16, 32]), train=rng.random() < 0.6)
    dtype = rng.choice(["f32", "bf16", "bf16", "f16"])
    D = rng.choice([32, 64, 64, 128]) if dtype == "f32" else rng.choice([64, 128])
    S = _length(rng, 48, 1536 if dtype == "f32" else 8192)
    T = S if rng.random() < 0.75 else _length(rng, 48, 1536 if dtype == "f32" else 8192)
    causal = S == T and rng.random() < 0.35
    B, H = _log_int(rng, 1, 32), rng.choice([1, 2, 4, 6, 8, 12, 16, 32])
    # the number of (query, key) pairs is kept below that of the listed cases
    limit = 3.0e8 if dtype == "f32" else 2.0e9
    while B * H * S * T > limit and B > 1:
        B = (B + 1) // 2
    while B * H * S * T > limit and H > 1:
        H = (H + 1) // 2
    bias, train = rng.choice(["none", "none", "full", "shared", "key"]), rng.random() < 0.7
    return _attention(None, dtype=dtype, B=B, H=H, S=S, T=T, D=D, train=train, bias=bias,
                      bias_grad=train and bias != "none" and rng.random() < 0.5, mask=rng.choice(["none", "none", "key", "full"]),
                      causal=causal, qk_norm=rng.random() < 0.15)


# ---- inputs ------------------------------------------------------------------------------------------------------
def _randn(g, shape, dtype, std=1.0):
    if len(shape) == 4 and math.prod(shape) > 1 << 28:      # bounded fp32 temporaries
        out = torch.empty(shape, device="cuda", dtype=dtype)
        for part in out:
            part.copy_(torch.randn(part.shape, generator=g, device="cuda") * std)
        return out
    return (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)


def _key_lengths(B, T):
    """Kept key counts of a padded batch, evenly spaced from T / 8 to T."""
    return [max(1, round(T * (1 / 8 + 7 / 8 * (i + 1) / B))) for i in range(B)]


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = _DTYPES[case["dtype"]]
    if case["op"] == "layer_norm":
        x = _randn(g, (case["rows"], case["C"]), dt)
        w = (1.0 + 0.1 * torch.randn(case["C"], generator=g, device="cuda")).to(dt)
        b = _randn(g, (case["C"],), dt, 0.1)
        state = dict(op="layer_norm", x=x, w=w, b=b, dy=None)
        if case["train"]:
            state["dy"] = _randn(g, (case["rows"], case["C"]), dt)
            for t in (x, w, b):
                t.requires_grad_(True)
        return state
    if case["op"] == "selective_scan":
        B, L, C, N = case["B"], case["L"], case["C"], case["N"]
        x = _randn(g, (B, L, C), dt)
        delta = (torch.rand((B, L, C), generator=g, device="cuda") * 0.5 + 0.01).to(dt)
        A = (-(torch.rand((C, N), generator=g, device="cuda") * 1.5 + 0.2)).to(dt)
        args = [x, delta, A, _randn(g, (B, L, N), dt), _randn(g, (B, L, N), dt), _randn(g, (C,), dt)]
        state = dict(op="selective_scan", args=args, dy=None)
        if case["train"]:
            state["dy"] = _randn(g, (B, L, C), dt)
            for t in args:
                t.requires_grad_(True)
        return state
    B, H, S, T, D = (case[n] for n in ("B", "H", "S", "T", "D"))
    q, k, v = _randn(g, (B, H, S, D), dt), _randn(g, (B, H, T, D), dt), _randn(g, (B, H, T, D), dt)
    bias = mask = None
    if case["bias"] == "full":
        bias = _randn(g, (B, H, S, T), dt, 0.5)
    elif case["bias"] == "key":
        bias = _randn(g, (1, H, 1, T), dt)
    elif case["bias"] == "shared":
        # a distance penalty per head plus what training has added to it
        slopes = torch.pow(2.0, -8.0 * (torch.arange(H, device="cuda", dtype=torch.float32) + 1) / H)
        dist = (torch.arange(S, device="cuda")[:, None] - torch.arange(T, device="cuda")[None, :]).abs().float()
        bias = torch.empty((1, H, S, T), device="cuda", dtype=dt)
        for h in range(H):
            bias[0, h] = (-slopes[h] * dist + 0.1 * torch.randn((S, T), generator=g, device="cuda")).to(dt)
    if case["mask"] == "key":
        # dealt to the batch in an order that the seed decides
        lens = torch.tensor(_key_lengths(B, T), device="cuda")[torch.randperm(B, generator=g, device="cuda")]
        mask = (torch.arange(T, device="cuda")[None, :] < lens[:, None]).reshape(B, 1, 1, T)
    elif case["mask"] == "full":
        mask = torch.rand((B, 1, S, T), generator=g, device="cuda") >= 0.1
        mask[..., 0] = True                                  # no row is left without a key, under causal as well
    state = dict(op="attention", q=q, k=k, v=v, bias=bias, mask=mask, causal=case["causal"], qk_norm=case["qk_norm"],
                 dout=None, leaves=None)
    if case["train"]:
        state["dout"] = _randn(g, (B, H, S, D), dt)
        state["leaves"] = [q, k, v] + ([bias] if case["bias_grad"] else [])
        for t in state["leaves"]:
            t.requires_grad_(True)
    return state


# ---- one pass ------------------------------------------------------------------------------------------------------
def run(state):
    if state["op"] == "layer_norm":
        y = layer_norm(state["x"], state["w"], state["b"])
        if state["dy"] is None:
            return [y]
        return [y.detach(), *torch.autograd.grad(y, [state["x"], state["w"], state["b"]], state["dy"])]
    if state["op"] == "selective_scan":
        y = selective_scan(*state["args"])
        if state["dy"] is None:
            return [y]
        return [y.detach(), *torch.autograd.grad(y, state["args"], state["dy"])]
    out = scaled_dot_product_attention(state["q"], state["k"], state["v"], bias=state["bias"], mask=state["mask"],
                                       causal=state["causal"], qk_norm=state["qk_norm"])
    if state["dout"] is None:
        return [out]
    return [out.detach(), *torch.autograd.grad(out, state["leaves"], state["dout"])]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def work(case):
    esz = _BYTES[case["dtype"]]
    if case["op"] == "layer_norm":
        n = case["rows"] * case["C"]
        if not case["train"]:
            return {"bytes": 2 * n * esz, "flops": 7 * n}
        return {"bytes": (2 + 3) * n * esz, "flops": 20 * n}   # x -> y; x, dy -> dx
    if case["op"] == "selective_scan":
        n, u = case["B"] * case["L"] * case["C"], case["B"] * case["L"] * case["C"] * case["N"]
        bc = 2 * case["B"] * case["L"] * case["N"]
        if not case["train"]:
            return {"bytes": (3 * n + bc) * esz, "flops": 7 * u}
        return {"bytes": (3 * n + bc + 5 * n + 2 * bc) * esz, "flops": (7 + 7 + 15) * u}
    B, H, S, T, D = (case[n] for n in ("B", "H", "S", "T", "D"))
    pairs = float(B * H) * S * T
    if case["mask"] == "key":
        pairs = float(H) * S * sum(_key_lengths(B, T))
    if case["causal"]:
        pairs *= 0.5 * (1.0 + 1.0 / S)
    q, kv = B * H * S * D * esz, B * H * T * D * esz
    bias = {"none": 0, "full": B * H * S * T, "shared": H * S * T, "key": H * T}[case["bias"]] * esz
    mask = {"none": 0, "full": B * S * T, "key": B * T}[case["mask"]]
    fwd = q + 2 * kv + q + bias + mask
    if not case["train"]:
        return {"bytes": int(fwd), "flops": int(4 * pairs * D)}
    bwd = 3 * q + 2 * kv + bias + mask + q + 2 * kv + (bias if case["bias_grad"] else 0)
    return {"bytes": int(fwd + bwd), "flops": int(14 * pairs * D)}


def tolerance(case):
    """Largest relative error (2-norm) of another correct implementation at the same precision: about four times what
    the outputs and gradients of each operation showed against its formula in 64 bits, over the listed shapes and forty
    drawn ones -- attention 8.8e-6 (fp32) / 4.1e-3 (bf16) / 4.2e-4 (fp16), LayerNorm 1.4e-7 / 1.8e-3 / 2.1e-4, scan
    7.2e-7 / 1.7e-3 / 2.1e-4."""
    return {"rel": {
        "attention": {"f32": 3e-5, "bf16": 1.6e-2, "f16": 2e-3},
        "layer_norm": {"f32": 1e-6, "bf16": 7e-3, "f16": 8.5e-4},
        "selective_scan": {"f32": 3e-6, "bf16": 7e-3, "f16": 8.5e-4},
    }[case["op"]][case["dtype"]]}
