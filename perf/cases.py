"""Workloads of the causal attention operator, from one short prompt to a full training step.

Every case goes through the public entry point :func:`flash_attention_v2`: ``forward`` cases call it
under ``no_grad`` (scoring or prefilling a prompt), ``train`` cases run it and its backward and return
the output together with the gradients.  A case holds

* ``direction``: ``forward`` or ``train``;
* ``batch``, ``heads``, ``seqlen``, ``headdim``;
* ``dtype``: ``fp16``, ``bf16`` or ``fp32`` (which the operator casts to fp16);
* ``layout``: ``dense`` (separate ``[B, H, N, D]`` tensors), ``rows`` (``[B, N, H, D]`` projections
  seen through a transpose) or ``packed`` (one ``[B, N, 3, H, D]`` projection);
* ``deterministic``, and optionally ``scale`` (0: the default ``1 / sqrt(headdim)``) and ``peak`` (the
  standard deviation of q and k; 1 unless given).
"""

from __future__ import annotations

import math

import torch

from flash_attention_triton_b200 import flash_attention_v2

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
#: what the largest listed case costs, in multiply-adds times two at the head dim the work is done at
_MOST_FLOPS = 3.85e12
_MOST_ELEMENTS = 2 * 32 * 8192 * 128


def _case(name, direction, batch, heads, seqlen, headdim, dtype, layout="dense", deterministic=False,
          scale=0.0, peak=1.0):
    return {"name": name, "direction": direction, "batch": batch, "heads": heads, "seqlen": seqlen,
            "headdim": headdim, "dtype": dtype, "layout": layout, "deterministic": deterministic,
            "scale": scale, "peak": peak}


def listed():
    return [
        # one short prompt through one layer: the time of a call, not of its arithmetic
        _case("prompt_128", "forward", 1, 8, 128, 64, "bf16"),
        # the smallest training step: unit tests, toy models, reproducible runs
        _case("train_256_det", "train", 2, 4, 256, 64, "fp16", deterministic=True),
        # a small language model on texts of about 1 000 tokens, projections packed as one tensor
        _case("train_1000_packed", "train", 8, 16, 1000, 64, "bf16", layout="packed"),
        # head dim 64 at an ordinary length, in both settings of the dQ summation
        _case("train_2048", "train", 4, 16, 2048, 64, "fp16"),
        _case("train_2048_det", "train", 4, 16, 2048, 64, "fp16", deterministic=True),
        # full-precision tensors handed over as they are, a head dim between the powers of two
        _case("train_1024_d96_fp32", "train", 32, 20, 1024, 96, "fp32"),
        # narrow heads, a ragged length, a peaked softmax with its own scale
        _case("train_4095_d32_det", "train", 8, 12, 4095, 32, "fp16", deterministic=True, scale=0.5,
              peak=3.0),
        # the main training shape of today's models
        _case("train_8192", "train", 2, 32, 8192, 128, "bf16"),
        # long context, the heads one GPU of a tensor-parallel group holds
        _case("train_32768", "train", 1, 2, 32768, 128, "bf16"),
        # the widest heads
        _case("train_8192_d256", "train", 2, 16, 8192, 256, "bf16"),
        # prefilling one long prompt
        _case("prefill_4096", "forward", 1, 32, 4096, 128, "bf16", layout="rows"),
        # scoring a few long documents with a head dim 64 model
        _case("prefill_8192_d64", "forward", 2, 16, 8192, 64, "fp16"),
    ]


def _pairs(seqlen):
    return seqlen * (seqlen + 1) // 2  # (query, key) pairs the causal mask keeps


def _cost(case):
    """Multiply-adds times two, head dims counted as 128 or 256 so that narrow heads, where the
    exponentials and not the products take the time, are not drawn larger than the listed ones."""
    wide = 128 if case["headdim"] <= 128 else 256
    passes = 1.0 if case["direction"] == "forward" else 3.5
    return passes * 4 * case["batch"] * case["heads"] * _pairs(case["seqlen"]) * wide


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    while True:
        direction = rng.choice(["train", "train", "forward"])
        seqlen = _log_uniform(rng, 64, 32768)
        if rng.random() < 0.5:
            seqlen = max(64, seqlen // 64 * 64)  # lengths people choose; the others come as they are
        headdim = rng.choice([32, 40, 48, 64, 64, 64, 80, 96, 128, 128, 128, 128, 160, 192, 256])
        dtype = rng.choice(["fp16", "fp16", "bf16", "bf16", "bf16", "fp32"])
        layout = rng.choice(["dense", "dense", "rows", "packed"])
        peaked = rng.random() < 0.15
        case = {"direction": direction, "batch": _log_uniform(rng, 1, 64), "heads": _log_uniform(rng, 1, 64),
                "seqlen": seqlen, "headdim": headdim, "dtype": dtype, "layout": layout,
                "deterministic": rng.random() < 0.35, "scale": 0.5 if peaked else 0.0,
                "peak": 3.0 if peaked and headdim <= 64 else 1.0}
        elements = case["batch"] * case["heads"] * seqlen * headdim
        if _cost(case) <= _MOST_FLOPS and elements <= _MOST_ELEMENTS:
            return case


def prepare(case, seed):
    b, h, n, d = (case[key] for key in ("batch", "heads", "seqlen", "headdim"))
    dtype = _DTYPES[case["dtype"]]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g, dtype=dtype)

    train = case["direction"] == "train"
    state = {"case": case, "scale": case["scale"] or None}
    if case["layout"] == "packed":
        qkv = normal(b, n, 3, h, d)
        if case["peak"] != 1.0:
            qkv[:, :, :2] *= case["peak"]
        state["leaves"] = [qkv]
    else:
        shape = (b, h, n, d) if case["layout"] == "dense" else (b, n, h, d)
        state["leaves"] = [normal(*shape) for _ in range(3)]
        if case["peak"] != 1.0:
            for t in state["leaves"][:2]:
                t *= case["peak"]
    if train:
        for t in state["leaves"]:
            t.requires_grad_(True)
        # the gradient arrives in the layout the model's next projection works in
        state["d_output"] = normal(b, h, n, d) if case["layout"] == "dense" else normal(b, n, h, d).transpose(1, 2)
    return state


def _q_k_v(state):
    layout, leaves = state["case"]["layout"], state["leaves"]
    if layout == "dense":
        return leaves
    if layout == "rows":
        return [t.transpose(1, 2) for t in leaves]
    return leaves[0].permute(2, 0, 3, 1, 4).unbind(0)


def run(state):
    case = state["case"]
    if case["direction"] == "forward":
        with torch.no_grad():
            q, k, v = _q_k_v(state)
            return flash_attention_v2(q, k, v, state["scale"], case["deterministic"])
    q, k, v = _q_k_v(state)
    out = flash_attention_v2(q, k, v, state["scale"], case["deterministic"])
    grads = torch.autograd.grad(out, state["leaves"], state["d_output"])
    return [out.detach(), *grads]


def work(case):
    """Causal attention over the pairs the mask keeps: two products of 2 d operations per pair forward
    and five backward; q, k, v (and dO) read once, O (and dq, dk, dv) written once."""
    b, h, n, d = (case[key] for key in ("batch", "heads", "seqlen", "headdim"))
    train = case["direction"] == "train"
    element = 4 if case["dtype"] == "fp32" else 2
    tensors = 8 if train else 4
    return {"bytes": tensors * b * h * n * d * element,
            "flops": (14 if train else 4) * b * h * _pairs(n) * d}


def tolerance(case):
    """Four times the error measured against the same formulas in fp64, on the listed cases and fourteen
    drawn ones: relative to the tensor's norm 3.4e-4 at fp16 and 2.9e-3 at bf16 whatever the size, and
    three times that with the peaked softmax; the largest single error, relative to the tensor's root
    mean square, grows with the length (the first rows' gradients are the largest): bf16 0.022 at 64,
    0.05 at 832, 0.13 at 8192 and 0.15 at 32768 rows, fp16 about a fifth of that, peaked twice."""
    bf16, peaked = case["dtype"] == "bf16", case["scale"] != 0.0
    largest = 0.1 * (case["seqlen"] / 64) ** 0.3
    return {"rel": (0.011 if bf16 else 0.0014) * (2.7 if peaked else 1.0),
            "max": min(0.9, (largest if bf16 else largest / 5) * (2.0 if peaked else 1.0))}
