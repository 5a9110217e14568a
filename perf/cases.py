"""What the framework's speed is measured on: its main paths through their public entry points, on one GPU.

Five kinds of work, over the sizes at which the configurations, tests and benchmark of this repository run them:

``tp_mlp``     forward of the tensor-parallel MLP block (``models.TPMLPBlock``), the headline configuration
``linear``     a linear layer (``ops.linear_bf16``), alone as in decoding or with its two gradients as in training
``attention``  flash attention (``ops.attention``), alone as in prefill or with its backward as in training
``moe``        forward of the expert-parallel MoE layer (``models.moe_layer.EPMoELayer``) with its three wire / expert precisions
``llama``      one training step of the FSDP decoder (``models.llama.FSDPLlama``): forward, backward, gradient exchange, optimiser

A case is a dict of plain values. ``prepare`` makes what a program holds before the call, ``run`` is one pass of the call.
"""
from __future__ import annotations

import dataclasses
import math

import torch

_context = None


def _ctx():
    """The process's distributed context (one rank), made once as a program does at its start."""
    global _context
    if _context is None:
        from parallelkernelbench_b200.parallel import init_context

        _context = init_context()
    return _context


class _Job:
    """One job's context with a symmetric heap of its own size, given back when the job is dropped."""

    def __init__(self, heap_bytes: int):
        from parallelkernelbench_b200.parallel.symm_heap import SymmetricHeap

        self.ctx = dataclasses.replace(_ctx(), owns_group=False, _heap=None)
        self.ctx._heap = SymmetricHeap.create(self.ctx, nbytes=int(heap_bytes) + (32 << 20))

    def __del__(self):
        try:
            self.ctx.finalize()
        except Exception:
            pass


# ------------------------------------------------------------------------------------------------ the cases
def listed() -> list[dict]:
    return [
        # one row block of a small block: what a call costs when the arithmetic is next to nothing
        {"name": "tp_mlp_small", "kind": "tp_mlp", "rows": 256, "hidden": 1024, "ffn": 4096},
        # the headline configuration at one rank
        {"name": "tp_mlp_block", "kind": "tp_mlp", "rows": 2048, "hidden": 8192, "ffn": 28672},
        # decoding: a batch of 16 tokens through the up projection of a 4096 / 14336 layer, bound by reading the weight
        {"name": "linear_decode", "kind": "linear", "tokens": 16, "k": 4096, "n": 14336, "act": "none", "bias": False, "train": False},
        # training on a ragged batch: forward with bias, dX and dW
        {"name": "linear_train_ragged", "kind": "linear", "tokens": 1333, "k": 4096, "n": 4104, "act": "none", "bias": True, "train": True},
        # the default attention configuration of the workloads, forward and backward
        {"name": "attn_train_1k", "kind": "attention", "b": 2, "s": 1024, "hq": 8, "hkv": 2, "d": 128, "causal": True, "train": True},
        # prefill of an odd length at head dimension 64, without a mask
        {"name": "attn_prefill_d64", "kind": "attention", "b": 1, "s": 3001, "hq": 32, "hkv": 8, "d": 64, "causal": False, "train": False},
        # long-context training: the sequence length and heads of the ring-attention configuration, one rank's share
        {"name": "attn_train_16k", "kind": "attention", "b": 1, "s": 16384, "hq": 32, "hkv": 8, "d": 128, "causal": True, "train": True},
        # the default MoE configuration: small experts, the data movement and the launches decide
        {"name": "moe_default", "kind": "moe", "tokens": 1024, "hidden": 1024, "inter": 128, "experts": 8, "topk": 2, "precision": "bf16"},
        # 7168 / 2048 experts, top-8, 8192 tokens per rank: 32 experts are one rank's share of the 256-expert configuration
        {"name": "moe_large_fp8_wire", "kind": "moe", "tokens": 8192, "hidden": 7168, "inter": 2048, "experts": 32, "topk": 8, "precision": "fp8_wire"},
        {"name": "moe_large_fp8_experts", "kind": "moe", "tokens": 8192, "hidden": 7168, "inter": 2048, "experts": 32, "topk": 8, "precision": "fp8_experts"},
        # a training step of the default decoder configuration: many small launches
        {"name": "llama_step_small", "kind": "llama", "layers": 2, "hidden": 512, "ffn": 1024, "heads": 4, "kv_heads": 2, "vocab": 8192, "seq": 256},
        # a training step of two layers, embedding and head of the 8B-shaped decoder
        {"name": "llama_step_8b_2layers", "kind": "llama", "layers": 2, "hidden": 4096, "ffn": 14336, "heads": 32, "kv_heads": 8, "vocab": 128256, "seq": 4096},
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_any(rng) -> dict:
    kind = rng.choice(["tp_mlp", "linear", "attention", "moe", "llama"])
    if kind == "tp_mlp":      # rows per rank come in 256s, the widths in 64s
        return {"kind": kind, "rows": 256 * _log_int(rng, 1, 16), "hidden": 64 * _log_int(rng, 8, 128), "ffn": 64 * _log_int(rng, 16, 448)}
    if kind == "linear":      # any number of tokens; the widths are multiples of 8 (the entry points ask for it)
        train = rng.random() < 0.5
        return {"kind": kind, "tokens": _log_int(rng, 1, 8192), "k": 8 * _log_int(rng, 32, 2048), "n": 8 * _log_int(rng, 32, 2048),
                "act": "none" if train else rng.choice(["none", "silu"]), "bias": rng.random() < 0.5, "train": train}
    if kind == "attention":
        hkv = rng.choice([1, 2, 4, 8])
        return {"kind": kind, "b": rng.choice([1, 1, 2, 4]), "s": _log_int(rng, 64, 16384), "hq": hkv * rng.choice([1, 2, 4]), "hkv": hkv,
                "d": rng.choice([64, 128]), "causal": rng.random() < 0.7, "train": rng.random() < 0.5}
    if kind == "moe":
        return {"kind": kind, "tokens": _log_int(rng, 16, 8192), "hidden": 128 * _log_int(rng, 4, 56), "inter": 128 * _log_int(rng, 1, 16),
                "experts": rng.choice([8, 16, 32, 64]), "topk": rng.choice([1, 2, 4, 8]), "precision": rng.choice(["bf16", "fp8_wire", "fp8_experts"])}
    kv, d = rng.choice([1, 2, 4, 8]), rng.choice([64, 128])
    heads = kv * rng.choice([1, 2, 4])
    heads = max(heads, 256 // d)
    return {"kind": "llama", "layers": rng.choice([1, 2]), "hidden": heads * d, "ffn": 128 * _log_int(rng, 4, 112), "heads": heads, "kv_heads": kv,
            "vocab": 8 * _log_int(rng, 512, 16032), "seq": _log_int(rng, 64, 4096)}


def draw(rng) -> dict:
    """One more case of the same ranges, at most as large as the largest listed one of its kind."""
    most = {}
    for c in listed():
        w = work(c)
        f, b = most.get(c["kind"], (0.0, 0.0))
        most[c["kind"]] = (max(f, w["flops"]), max(b, w["bytes"]))
    while True:
        c = _draw_any(rng)
        w = work(c)
        f, b = most[c["kind"]]
        if w["flops"] <= f and w["bytes"] <= max(b, 1 << 30):
            return c


# ------------------------------------------------------------------------------------------------ what a program holds
def _rand(shape, gen, std: float = 1.0) -> torch.Tensor:
    x = torch.randn(*shape, device="cuda", dtype=torch.float32, generator=gen)
    return (x.mul_(std) if std != 1.0 else x).to(torch.bfloat16)


def _prepare_tp_mlp(c, seed, gen):
    from parallelkernelbench_b200.models import TPMLPBlock, TPMLPConfig

    cfg = TPMLPConfig(rows_per_rank=c["rows"], hidden=c["hidden"], ffn=c["ffn"])
    job = _Job(4 * c["rows"] * c["hidden"])
    w1, w2, gamma = TPMLPBlock.random_weights(cfg, 1, 0, job.ctx.device, seed=seed)
    gamma.add_(_rand((c["hidden"],), gen, 0.1))
    return {"job": job, "block": TPMLPBlock(job.ctx.heap().world_group, cfg, w1, w2, gamma), "x": _rand((c["rows"], c["hidden"]), gen)}


def _prepare_linear(c, seed, gen):
    t, k, n = c["tokens"], c["k"], c["n"]
    s = {"x": _rand((t, k), gen), "w": _rand((n, k), gen, 0.02), "bias": _rand((n,), gen, 0.1) if c["bias"] else None, "act": c["act"]}
    s["dy"] = _rand((t, n), gen) if c["train"] else None
    return s


def _prepare_attention(c, seed, gen):
    b, s, d = c["b"], c["s"], c["d"]
    st = {"q": _rand((b, s, c["hq"], d), gen), "k": _rand((b, s, c["hkv"], d), gen), "v": _rand((b, s, c["hkv"], d), gen), "causal": c["causal"]}
    st["dout"] = _rand((b, s, c["hq"], d), gen) if c["train"] else None
    return st


def _prepare_moe(c, seed, gen):
    from parallelkernelbench_b200.models.moe_layer import EPMoELayer, MoEConfig
    from parallelkernelbench_b200.parallel.comm import Comm

    cfg = MoEConfig(hidden=c["hidden"], inter=c["inter"], num_experts=c["experts"], top_k=c["topk"], tokens_per_rank=c["tokens"],
                    fp8_dispatch=c["precision"] != "bf16", fp8_experts=c["precision"] == "fp8_experts")
    capacity = int(c["tokens"] * c["topk"] * cfg.capacity_factor + 127)
    job = _Job(capacity * (4 * c["hidden"] + 1024))
    weights = EPMoELayer.random_weights(cfg, 1, 0, job.ctx.device, seed=seed)
    bias = torch.randn(c["experts"], device="cuda", generator=gen) * 0.1
    layer = EPMoELayer(job.ctx.heap().world_group, Comm(job.ctx), cfg, *weights, router_bias=bias)
    return {"job": job, "layer": layer, "x": _rand((c["tokens"], c["hidden"]), gen)}


def _prepare_llama(c, seed, gen):
    from parallelkernelbench_b200.models.llama import FSDPLlama, LlamaConfig

    job = _Job(1 << 20)
    model = FSDPLlama(job.ctx, LlamaConfig(**{k: v for k, v in c.items() if k not in ("name", "kind")}))
    tokens = torch.randint(0, c["vocab"], (c["seq"] + 1,), device="cuda", generator=gen)
    return {"job": job, "model": model, "tokens": tokens[:-1].contiguous(), "targets": tokens[1:].contiguous()}


_PREPARE = {"tp_mlp": _prepare_tp_mlp, "linear": _prepare_linear, "attention": _prepare_attention, "moe": _prepare_moe, "llama": _prepare_llama}


def prepare(case: dict, seed: int) -> dict:
    _ctx()
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    return {"kind": case["kind"], **_PREPARE[case["kind"]](case, int(seed), gen)}


# ------------------------------------------------------------------------------------------------ one pass
def _run_linear(s):
    from parallelkernelbench_b200.ops import gemm_bf16_kn, gemm_bf16_tn, linear_bf16

    y = linear_bf16(s["x"], s["w"], bias=s["bias"], activation=s["act"])
    if s["dy"] is None:
        return {"y": y}
    return {"y": y, "dx": gemm_bf16_kn(s["dy"], s["w"]), "dw": gemm_bf16_tn(s["dy"], s["x"])}


def _run_attention(s):
    from parallelkernelbench_b200.ops.attention import flash_attn_bwd, flash_attn_fwd

    out, lse = flash_attn_fwd(s["q"], s["k"], s["v"], causal=s["causal"])
    if s["dout"] is None:
        return {"out": out, "lse": lse}
    dq, dk, dv = flash_attn_bwd(s["q"], s["k"], s["v"], out, lse, s["dout"], causal=s["causal"])
    return {"out": out, "lse": lse, "dq": dq, "dk": dk, "dv": dv}


def _run_llama(s):
    # loss and updated weights. The optimiser's moments are left out: the gradient is quantised to e4m3 (steps of 6 to 12 %) on its way to
    # them, and a bf16 rounding of another correct implementation moves 2 to 5 % of their norm across a step - more than can be told
    # from an error. The weights' update is +-lr wherever the sign of the gradient is right, and shows what they would.
    m = s["model"]
    out = {"loss": m.step(s["tokens"], s["targets"]), "head": m.head_master, "head_bf16": m.head.data, "embed": m.embed.master}
    out["layers"] = [u.master for u in m.units]
    return out


def run(state: dict):
    kind = state["kind"]
    if kind == "tp_mlp":
        return {"y": state["block"](state["x"])}
    if kind == "linear":
        return _run_linear(state)
    if kind == "attention":
        return _run_attention(state)
    if kind == "moe":
        return {"y": state["layer"](state["x"])}
    return _run_llama(state)


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case: dict) -> dict:
    c, kind = case, case["kind"]
    if kind == "tp_mlp":
        return {"flops": 4.0 * c["rows"] * c["hidden"] * c["ffn"], "bytes": 4.0 * c["hidden"] * c["ffn"] + 4.0 * c["rows"] * c["hidden"]}
    if kind == "linear":
        t, k, n = c["tokens"], c["k"], c["n"]
        if not c["train"]:
            return {"flops": 2.0 * t * k * n, "bytes": 2.0 * (t * k + n * k + t * n)}
        return {"flops": 6.0 * t * k * n, "bytes": 2.0 * (2 * t * k + 2 * n * k + 2 * t * n)}
    if kind == "attention":
        b, s, d, hq, hkv = c["b"], c["s"], c["d"], c["hq"], c["hkv"]
        pairs = 0.5 * s * (s + 1) if c["causal"] else float(s) * s
        q, kv, lse = b * s * hq * d, b * s * hkv * d, b * s * hq
        if not c["train"]:
            return {"flops": 4.0 * b * hq * d * pairs, "bytes": 2.0 * (2 * q + 2 * kv) + 4.0 * lse}
        return {"flops": 14.0 * b * hq * d * pairs, "bytes": 2.0 * (3 * q + 2 * kv) + 4.0 * (lse + q + 2 * kv)}
    if kind == "moe":
        t, h, i, e = c["tokens"], c["hidden"], c["inter"], c["experts"]
        return {"flops": 6.0 * t * c["topk"] * h * i + 2.0 * t * h * e,
                "bytes": 3.0 * e * h * i * (1 if c["precision"] == "fp8_experts" else 2) + 2.0 * e * h + 4.0 * t * h}
    d, s, h = c["hidden"] // c["heads"], c["seq"], c["hidden"]
    layer = (c["heads"] + 2 * c["kv_heads"]) * d * h + h * h + 3 * h * c["ffn"]
    flops = 6.0 * s * (c["layers"] * layer + c["vocab"] * h) + 14.0 * c["layers"] * h * 0.5 * s * (s + 1)
    # fp32 master and two moments read and written, one byte per parameter of the wire copy read and written (head: its bf16 copy)
    return {"flops": flops, "bytes": 26.0 * (c["layers"] * layer + c["vocab"] * h) + 28.0 * c["vocab"] * h}


def tolerance(case: dict):
    """About four times what was measured (relative error in the 2-norm / largest error over the root mean square or the value):
    linear, against 64 bits: 1.7e-3 / 4e-3 (the rounding of a bf16 result); attention, against 64 bits: 2.4e-3 / 6.5e-2 (bf16
    probabilities and their gradients); tp_mlp, against the same stages as library products: 4.1e-3 / 2.3e-2 (bf16 hidden
    activations and partial sums); moe against 64-bit products on the same routing: 2.9e-3 / 2.2e-2, with e4m3 experts 1.2e-2 / 0.14
    (single codes of the re-quantised activations); llama, one and two steps against the same step on library products and library
    attention: 1.7e-3 / 6.1e-2 on the weights."""
    kind = case["kind"]
    if kind == "moe" and case["precision"] == "fp8_experts":
        return {"rel": 3e-2, "max": 0.6}
    return {"linear": {"rel": 6e-3, "max": 2e-2}, "attention": {"rel": 1e-2, "max": 0.26}, "tp_mlp": {"rel": 1.2e-2, "max": 0.1},
            "moe": {"rel": 1.2e-2, "max": 0.1}, "llama": {"rel": 7e-3, "max": 0.25}}[kind]
