"""The work whose speed is measured: calls of the framework's public entry points, as model code makes them.

Two kinds of work make up a mixture-of-experts decoder: the mixture-of-experts block (one call per layer) and the
quantized projections around it.  Ops of a case:

  forward   `MoEMLP.forward_with_stream(x)`: the block, as prefill and an eager decode loop call it
  layer     `MoEMLP.forward_residual(h, norm)`: h + block(rms_norm(h)), the second half of a decoder layer
  replay    `MoEMLP.capture(x)` kept, then called with each step's activations: a decode loop with fixed shapes
  linear    `QuantizedLinear.forward_with_stream(x)`: attention projections and the vocabulary head

The layer shapes are those of `ironmlx_b200.workloads.CONFIGS` (hidden 2048, 256 experts of width 512, top-8, a
shared expert; and the small layer of 16 experts without one) and one between them.
"""
from __future__ import annotations

import math

import torch

from ironmlx_b200 import nn, ops
from ironmlx_b200.workloads import MoEConfig, algorithmic_bytes_decode, algorithmic_flops

# hidden, experts, experts per token, expert width, width of the shared expert (0: none)
LARGE = dict(hidden=2048, experts=256, top_k=8, width=512, shared=512)
MIDDLE = dict(hidden=1024, experts=64, top_k=4, width=512, shared=512)
SMALL = dict(hidden=512, experts=16, top_k=4, width=256, shared=0)

# mode, bits, group: every weight format that checkpoints come in, the usual group sizes first
AFFINE4 = dict(mode="affine", bits=4, group=64)
AFFINE2 = dict(mode="affine", bits=2, group=64)
AFFINE6 = dict(mode="affine", bits=6, group=64)
AFFINE8 = dict(mode="affine", bits=8, group=64)
MXFP8 = dict(mode="mxfp8", bits=8, group=32)
NVFP4 = dict(mode="nvfp4", bits=4, group=16)

_HOT_SHARE = 0.08        # skewed routing: share of the assignments that the most popular expert gets


def _moe(name, op, tokens, shape, fmt, skew=0.0):
    return dict(name=name, op=op, tokens=tokens, skew=skew, **shape, **fmt)


def _linear(name, rows, n_in, n_out, fmt):
    return dict(name=name, op="linear", rows=rows, n_in=n_in, n_out=n_out, **fmt)


def listed():
    return [
        # one user's decode step: latency and launches, a handful of experts' weights
        _moe("decode-1", "forward", 1, LARGE, AFFINE4),
        # a small batch of an odd size through the whole second half of a decoder layer
        _moe("decode-19-layer", "layer", 19, LARGE, AFFINE4),
        # the serving step with the layer's calls recorded once (the benchmark's decode workload)
        _moe("decode-64-replay", "replay", 64, LARGE, AFFINE4),
        # larger decode batches with block-scaled float weights
        _moe("decode-256-nvfp4", "forward", 256, LARGE, NVFP4),
        _moe("decode-256-mxfp8", "forward", 256, LARGE, MXFP8),
        # a width that does not divide a word: 6-bit checkpoints, a medium prompt
        _moe("prefill-1000-6bit", "forward", 1000, LARGE, AFFINE6),
        # a prompt of no round length, through the whole second half of a decoder layer
        _moe("prefill-1777-8bit-layer", "layer", 1777, LARGE, AFFINE8),
        # long prompts: the benchmark's prefill workload and the same with block-scaled fp4 weights
        _moe("prefill-8192", "forward", 8192, LARGE, AFFINE4),
        _moe("prefill-4096-nvfp4", "forward", 4096, LARGE, NVFP4),
        # the largest: skewed expert popularity, a few experts see most tokens
        _moe("prefill-16384-skew-2bit", "forward", 16384, LARGE, AFFINE2, skew=1.2),
        # the vocabulary head of a small decode batch, and an attention projection of a ragged prompt
        _linear("head-6", 6, 2048, 152064, AFFINE4),
        _linear("projection-777", 777, 2048, 8192, AFFINE4),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    fmt = dict(rng.choice([AFFINE4, AFFINE4, AFFINE4, AFFINE8, AFFINE2, MXFP8, NVFP4, AFFINE6,
                           dict(mode="affine", bits=3, group=64), dict(mode="affine", bits=5, group=64),
                           dict(mode="affine", bits=4, group=32), dict(mode="affine", bits=8, group=128)]))
    # the widths that do not divide a word, and groups of 32, come with short and medium prompts
    short = fmt["bits"] in (3, 5, 6) or (fmt["mode"] == "affine" and fmt["group"] == 32)
    if rng.random() < 0.25:
        n_in, n_out = rng.choice([(512, 2048), (1024, 1024), (2048, 512), (2048, 4096), (2048, 8192), (4096, 2048),
                                  (2048, 152064)])
        most = 64 if n_out > 100000 else 8192
        if short:
            most = min(most, int(4e10 / (2.0 * n_in * n_out)))
        return dict(op="linear", rows=_log_uniform(rng, 1, most), n_in=n_in, n_out=n_out, **fmt)
    shape = rng.choice([LARGE, LARGE, LARGE, MIDDLE, SMALL])
    tokens = _log_uniform(rng, 1, 1000 if short else 16384)
    if tokens <= 256:
        op = rng.choice(["forward", "layer", "replay"])
    else:
        op = rng.choice(["forward", "layer"])
    skew = 1.2 if tokens >= 1024 and rng.random() < 0.3 else 0.0
    return dict(op=op, tokens=tokens, skew=skew, **shape, **fmt)


# ── inputs ──────────────────────────────────────────────────────────────────
def _normal(gen, *shape, std=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * std).to(torch.bfloat16)


def _quantized(gen, case, *shape):
    """Weights ~N(0, 0.02) in the case's format."""
    w = torch.randn(*shape, generator=gen, device="cuda").mul_(0.02)
    q = ops.quantize(w, case["group"], case["bits"], case["mode"])
    return nn.QuantizedLinear(q[0], q[1], q[2], case["group"], case["bits"], case["mode"], q[3] if len(q) > 3 else None)


def _popularity_bias(gen, x, router, top_k, s):
    """Per-expert logit bias that makes expert popularity follow a Zipf law: a * log(1 / rank^s), a bisected on a
    sample of tokens until the most popular expert gets its share of the assignments."""
    experts = router.shape[0]
    rank = torch.randperm(experts, generator=gen, device="cuda").float() + 1.0
    logw = -s * torch.log(rank)
    z = x[:2048].float() @ router.float().T
    lo, hi = 0.0, 8.0
    for _ in range(20):
        mid = 0.5 * (lo + hi)
        top = torch.topk(z + mid * logw, top_k, dim=-1).indices.reshape(-1)
        if torch.bincount(top, minlength=experts).max().item() < _HOT_SHARE * top.numel():
            lo = mid
        else:
            hi = mid
    return (0.5 * (lo + hi) * logw).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["op"] == "linear":
        return {"op": "linear", "layer": _quantized(gen, case, case["n_out"], case["n_in"]),
                "x": _normal(gen, case["rows"], case["n_in"])}
    h, e, w, sh = case["hidden"], case["experts"], case["width"], case["shared"]
    x = _normal(gen, case["tokens"], h)
    router = _normal(gen, e, h, std=0.02)
    experts = nn.FusedExperts(_quantized(gen, case, e, 2 * w, h), _quantized(gen, case, e, h, w))
    shared = shared_gate = None
    if sh:
        shared = nn.MLP(_quantized(gen, case, sh, h), _quantized(gen, case, sh, h), _quantized(gen, case, h, sh))
        shared_gate = nn.Linear(_normal(gen, 1, h, std=0.02))
    bias = _popularity_bias(gen, x, router, case["top_k"], case["skew"]) if case["skew"] else None
    moe = nn.MoEMLP(nn.Linear(router), experts, shared, shared_gate, case["top_k"], True, bias)
    state = {"op": case["op"], "moe": moe, "x": x}
    if case["op"] == "layer":
        state["norm"] = nn.RMSNorm.new(_normal(gen, h, std=0.1) + 1.0, 1e-6)
    elif case["op"] == "replay":
        state["step"] = moe.capture(torch.zeros_like(x))
    return state


def run(state):
    if state["op"] == "linear":
        return state["layer"].forward_with_stream(state["x"])
    if state["op"] == "layer":
        return state["moe"].forward_residual(state["x"], state["norm"])
    if state["op"] == "replay":
        return state["step"](state["x"])
    return state["moe"].forward_with_stream(state["x"])


# ── what a pass cannot do without ───────────────────────────────────────────
def _weight_bytes(case):
    per = {"affine": case["bits"] / 8 + 4 / case["group"], "mxfp8": 1 + 1 / 32, "nvfp4": 0.5 + 1 / 16}
    return per[case["mode"]]


def work(case):
    if case["op"] == "linear":
        m, k, n = case["rows"], case["n_in"], case["n_out"]
        return {"bytes": n * k * _weight_bytes(case) + 2 * m * (k + n), "flops": 2 * m * k * n}
    cfg = MoEConfig("case", tokens=case["tokens"], hidden=case["hidden"], num_experts=case["experts"],
                    top_k=case["top_k"], intermediate=case["width"], shared_intermediate=case["shared"],
                    mode=case["mode"], bits=case["bits"], group_size=case["group"])
    # experts that at least one token picks, with uniform routing (a skewed router picks no more)
    touched = case["experts"] * (1.0 - (1.0 - case["top_k"] / case["experts"]) ** case["tokens"])
    return {"bytes": algorithmic_bytes_decode(cfg, int(round(touched))), "flops": algorithmic_flops(cfg)}


def tolerance(case):
    """Against fp64 the outputs are 1.66e-3 off (2-norm), nearly all of it the one rounding to bf16, and 4.3e-3 at
    the most for a single value: four times that is stated.  A block over many tokens meets rows whose k-th and
    next expert's logits agree to the last bits of an fp32 sum (about one row in 50 000): such a row may take the
    other expert, which moves single values by up to 0.9 and hardly shows in the norm."""
    if case["op"] == "linear":
        return {"rel": 6.7e-3, "max": 0.02}
    return {"rel": 6.7e-3, "max": 0.9 if case["tokens"] >= 512 else 0.02}
