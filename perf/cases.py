"""The workloads this library is timed on, on one GPU: every public path that a serving or training
program calls, over the sizes it calls them with.

``listed()`` names the standing cases and ``draw(rng)`` gives one more of the same ranges; ``prepare``
builds what a program holds before the call (a context, a layer, weights, inputs made from the seed),
``run`` is one pass through the public entry points, ``work`` counts the bytes and operations that the
pass cannot do without and ``tolerance`` says how far two correct implementations may lie apart.

Layers are shared by all states of one configuration, as a program keeps one layer and feeds it new
inputs; a layer's context is closed when the last state that uses it is gone.
"""
from __future__ import annotations

import json
import math
import weakref

import torch
import torch.distributed as dist

import iris_b200 as iris
from iris_b200.models import FlashDecodeLayer, MoELayer, RingAttention, TensorParallelMLP
from iris_b200.ops import all_gather_matmul_preamble, matmul, matmul_reduce_scatter_preamble, quantize_activation, quantize_weight

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
HEAD_DIM = 128


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # a linear layer of a decode step: 16 tokens through the 8-way tensor-parallel slice of an up projection
        {"name": "gemm_decode", "kind": "gemm", "tokens": 16, "out": 3584, "in": 8192, "layout": "linear", "bias": False, "dtype": "bf16"},
        # a prompt of no round length through a projection stored (in, out), with bias
        {"name": "gemm_prompt", "kind": "gemm", "tokens": 1000, "out": 8192, "in": 3584, "layout": "row", "bias": True, "dtype": "fp16"},
        # the same slice in e4m3: activations quantised on the fly, weights quantised at load time
        {"name": "linear_e4m3", "kind": "linear_e4m3", "tokens": 4096, "out": 3584, "in": 8192, "dtype": "bf16"},
        # tensor-parallel MLP in inference (gather, up, down, scatter): a decode step and a full prefill batch
        {"name": "tp_mlp_decode", "kind": "tp_mlp", "tokens": 48, "hidden": 8192, "ffn": 3584, "dtype": "bf16"},
        {"name": "tp_mlp_prefill", "kind": "tp_mlp", "tokens": 8192, "hidden": 8192, "ffn": 3584, "dtype": "bf16"},
        # one training step of the same layer: forward and backward, gradients of the input and both weights
        {"name": "tp_mlp_train", "kind": "tp_mlp_train", "tokens": 2048, "hidden": 8192, "ffn": 3584, "activation": "silu", "dtype": "bf16"},
        # mixture of experts: a decode batch in e4m3 (bound by the expert weights) and a prefill batch in bf16
        {"name": "moe_decode", "kind": "moe", "tokens": 64, "hidden": 7168, "ffn": 2048, "experts": 32, "top_k": 8, "e4m3": True},
        {"name": "moe_prefill", "kind": "moe", "tokens": 4096, "hidden": 7168, "ffn": 2048, "experts": 32, "top_k": 8, "e4m3": False},
        # attention of a decode step: one long sequence (latency), and a ragged batch
        {"name": "decode_single", "kind": "decode", "batch": 1, "length": 32768, "shortest": 32768, "q_heads": 64, "kv_heads": 8,
         "page": 64, "soft_cap": 0.0, "dtype": "bf16"},
        {"name": "decode_batch", "kind": "decode", "batch": 32, "length": 32768, "shortest": 8192, "q_heads": 64, "kv_heads": 8,
         "page": 16, "soft_cap": 0.0, "dtype": "bf16"},
        # attention of a prefill: a causal block of a long context, and a full-attention one of no round length
        {"name": "attention_causal", "kind": "attention", "tokens": 8192, "q_heads": 32, "kv_heads": 8, "causal": True, "dtype": "bf16"},
        {"name": "attention_ragged", "kind": "attention", "tokens": 3000, "q_heads": 32, "kv_heads": 8, "causal": False, "dtype": "fp16"},
    ]


def _log_int(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    while True:
        kind = rng.choice(["gemm", "linear_e4m3", "tp_mlp", "tp_mlp_train", "moe", "decode", "attention"])
        if kind == "gemm":
            case = {"kind": kind, "tokens": _log_int(rng, 1, 8192), "out": 8 * _log_int(rng, 128, 1024), "in": 8 * _log_int(rng, 128, 1024),
                    "layout": rng.choice(["linear", "linear", "row"]), "bias": rng.random() < 0.4, "dtype": dtype}
        elif kind == "linear_e4m3":
            case = {"kind": kind, "tokens": _log_int(rng, 1, 8192), "out": 64 * _log_int(rng, 16, 128), "in": 128 * _log_int(rng, 8, 64), "dtype": dtype}
        elif kind == "tp_mlp":
            tokens = _log_int(rng, 1, 8192)
            if rng.random() < 0.5:
                tokens = -(-tokens // 128) * 128
            case = {"kind": kind, "tokens": tokens, "hidden": 256 * _log_int(rng, 4, 32), "ffn": 128 * _log_int(rng, 4, 28), "dtype": dtype}
        elif kind == "tp_mlp_train":
            case = {"kind": kind, "tokens": 128 * _log_int(rng, 1, 32), "hidden": 256 * _log_int(rng, 4, 32), "ffn": 128 * _log_int(rng, 4, 28),
                    "activation": rng.choice(["silu", "silu", "gelu"]), "dtype": dtype}
        elif kind == "moe":
            case = {"kind": kind, "tokens": _log_int(rng, 1, 4096), "hidden": rng.choice([1024, 2048, 4096, 5120, 7168]),
                    "ffn": rng.choice([512, 768, 1024, 1408, 2048]), "experts": rng.choice([8, 16, 32, 64]), "top_k": rng.choice([2, 4, 6, 8]),
                    "e4m3": rng.random() < 0.5}
        elif kind == "decode":
            kv_heads = rng.choice([2, 4, 8])
            length = _log_int(rng, 256, 131072)
            case = {"kind": kind, "batch": _log_int(rng, 1, 64), "length": length, "shortest": rng.choice([length, max(1, length // 4), max(1, length // 16)]),
                    "q_heads": kv_heads * rng.choice([1, 4, 8]), "kv_heads": kv_heads, "page": rng.choice([16, 32, 64, 128]),
                    "soft_cap": rng.choice([0.0, 0.0, 30.0]), "dtype": dtype}
        else:
            tokens = _log_int(rng, 128, 8192)
            if rng.random() < 0.5:
                tokens = -(-tokens // 128) * 128
            kv_heads = rng.choice([2, 4, 8])
            case = {"kind": kind, "tokens": tokens, "q_heads": kv_heads * rng.choice([1, 2, 4]), "kv_heads": kv_heads,
                    "causal": rng.random() < 0.6, "dtype": dtype}
        w = work(case)
        cap = work(listed()[7])          # the largest listed case
        if w["flops"] <= cap["flops"] and w["bytes"] <= 1.2 * cap["bytes"] and _held(case) <= 6e9:
            return case


def _held(case):
    """Bytes of inputs that one state of a decode case holds (its cache is allocated for the longest length)."""
    if case["kind"] != "decode":
        return 0.0
    return 4.0 * case["batch"] * case["length"] * case["kv_heads"] * HEAD_DIM


# ---------------------------------------------------------------------------------------- prepare
def _rand(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))

    def normal(*shape, scale=1.0, dtype=torch.float32):
        return (torch.randn(*shape, device="cuda", generator=g, dtype=torch.float32) * scale).to(dtype)

    return g, normal


def _context(heap_bytes):
    if not dist.is_initialized():
        torch.cuda.set_device(0)
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
    return iris.iris(int(heap_bytes) + (128 << 20))


class _Handle:
    """A context and the layer that lives on it; the context is closed with the last state that uses it."""

    def __init__(self, heap_bytes):
        self.ctx = _context(heap_bytes)
        self.layer = None

    def __del__(self):
        ctx = self.__dict__.get("ctx")
        if ctx is not None:
            ctx.close()


_handles: "weakref.WeakValueDictionary[str, _Handle]" = weakref.WeakValueDictionary()


def _handle(case, make):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    h = _handles.get(key)
    if h is None:
        h = make()
        _handles[key] = h
    return h


def _make_tp(case):
    T, D = case["tokens"], case["hidden"]
    h = _Handle(24 * (T + 256) * max(D, case["ffn"]))
    if case["kind"] == "tp_mlp_train":
        _, normal = _rand(1)
        dt = DTYPES[case["dtype"]]
        h.layer = TensorParallelMLP(h.ctx, D, case["ffn"], activation=case["activation"], dtype=dt,
                                    w1=normal(D, case["ffn"], scale=D ** -0.5, dtype=dt), w2=normal(case["ffn"], D, scale=case["ffn"] ** -0.5, dtype=dt))
    return h


def _make_moe(case):
    T, D, F, E, K = (case[k] for k in ("tokens", "hidden", "ffn", "experts", "top_k"))
    rows = T * K + 128
    h = _Handle(4.5 * rows * D + 64 * rows)
    _, normal = _rand(2)
    bf = torch.bfloat16
    h.layer = MoELayer(h.ctx, D, F, E, K, max_tokens=T, w_gate=normal(E, D, F, scale=D ** -0.5, dtype=bf), w_up=normal(E, D, F, scale=D ** -0.5, dtype=bf),
                       w_down=normal(E, F, D, scale=F ** -0.5, dtype=bf), fp8=case["e4m3"])
    return h


def _make_decode(case):
    h = _Handle(8 * case["batch"] * case["q_heads"] * (HEAD_DIM + 2) * 2)
    h.layer = FlashDecodeLayer(h.ctx, case["q_heads"], case["kv_heads"], HEAD_DIM, max_batch=case["batch"], soft_cap=case["soft_cap"],
                               dtype=DTYPES[case["dtype"]])
    return h


def _make_attention(case):
    h = _Handle(8 * case["tokens"] * case["kv_heads"] * HEAD_DIM)
    h.layer = RingAttention(h.ctx, case["tokens"], case["q_heads"], case["kv_heads"], dtype=DTYPES[case["dtype"]])
    return h


def prepare(case, seed):
    g, normal = _rand(seed)
    kind = case["kind"]
    dt = DTYPES[case.get("dtype", "bf16")]
    s = {"kind": kind}
    if kind == "gemm":
        T, N, K = case["tokens"], case["out"], case["in"]
        s["x"] = normal(T, K, dtype=dt)
        s["w"] = normal(N, K, scale=K ** -0.5, dtype=dt).t() if case["layout"] == "linear" else normal(K, N, scale=K ** -0.5, dtype=dt)
        s["bias"] = normal(N, dtype=dt) if case["bias"] else None
    elif kind == "linear_e4m3":
        s["x"] = normal(case["tokens"], case["in"], dtype=dt)
        s["w"] = quantize_weight(normal(case["out"], case["in"], scale=case["in"] ** -0.5))
        s["out"] = torch.empty(case["tokens"], case["out"], dtype=dt, device="cuda")
    elif kind == "tp_mlp":
        T, D, F = case["tokens"], case["hidden"], case["ffn"]
        s["handle"] = h = _handle(case, lambda: _make_tp(case))
        s["x"] = normal(T, D, dtype=dt)
        s["w1"] = normal(F, D, scale=D ** -0.5, dtype=dt).t()
        s["w2"] = normal(D, F, scale=F ** -0.5, dtype=dt).t()
        s["h"] = torch.empty(T, F, dtype=dt, device="cuda")
        s["y"] = torch.empty(T, D, dtype=dt, device="cuda")
        if h.layer is None:
            h.layer = (all_gather_matmul_preamble(h.ctx, s["x"], s["w1"], shard_dim=0),
                       matmul_reduce_scatter_preamble(h.ctx, s["y"], s["h"], s["w2"], scatter_rows=True))
    elif kind == "tp_mlp_train":
        s["handle"] = _handle(case, lambda: _make_tp(case))
        s["x"] = normal(case["tokens"], case["hidden"], dtype=dt).requires_grad_(True)
        s["dy"] = normal(case["tokens"], case["hidden"], scale=case["tokens"] ** -0.5, dtype=dt)
    elif kind == "moe":
        s["handle"] = _handle(case, lambda: _make_moe(case))
        s["x"] = normal(case["tokens"], case["hidden"], dtype=torch.bfloat16)
        # some experts are more popular than others
        s["logits"] = normal(case["tokens"], case["experts"]) + normal(1, case["experts"], scale=0.5)
    elif kind == "decode":
        B, L, page, Hkv = case["batch"], case["length"], case["page"], case["kv_heads"]
        s["handle"] = _handle(case, lambda: _make_decode(case))
        blocks = -(-L // page)
        s["q"] = normal(B, case["q_heads"], HEAD_DIM, dtype=dt)
        cache = lambda: torch.empty(B * blocks, page, Hkv, HEAD_DIM, dtype=dt, device="cuda").normal_(generator=g)  # noqa: E731
        s["k"], s["v"] = cache(), cache()
        # the pages of a sequence lie anywhere in the cache
        s["table"] = torch.randperm(B * blocks, device="cuda", generator=g).to(torch.int32).view(B, blocks)
        s["lens"] = torch.randint(case["shortest"], L + 1, (1, B), device="cuda", generator=g, dtype=torch.int32)
    else:
        T = case["tokens"]
        s["handle"] = _handle(case, lambda: _make_attention(case))
        s["q"] = normal(T, case["q_heads"], HEAD_DIM, dtype=dt)
        s["k"] = normal(T, case["kv_heads"], HEAD_DIM, dtype=dt)
        s["v"] = normal(T, case["kv_heads"], HEAD_DIM, dtype=dt)
        s["causal"] = case["causal"]
    return s


# -------------------------------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "gemm":
        return matmul(s["x"], s["w"], bias=s["bias"])
    if kind == "linear_e4m3":
        return matmul(quantize_activation(s["x"]), s["w"], out=s["out"])
    if kind == "tp_mlp":
        ctx, (up, down) = s["handle"].ctx, s["handle"].layer
        ctx.ops.all_gather_matmul(s["h"], s["x"], s["w1"], shard_dim=0, workspace=up, async_op=True)
        ctx.ops.matmul_reduce_scatter(s["y"], s["h"], s["w2"], scatter_rows=True, workspace=down, async_op=True)
        return s["h"], s["y"]
    if kind == "tp_mlp_train":
        mlp, x = s["handle"].layer, s["x"]
        mlp.zero_grad(set_to_none=True)
        x.grad = None
        y = mlp(x)
        y.backward(s["dy"])
        return y.detach(), x.grad, mlp.w1.grad, mlp.w2.grad
    if kind == "moe":
        return s["handle"].layer(s["x"], s["logits"])
    if kind == "decode":
        return s["handle"].layer(s["q"], s["k"], s["v"], s["lens"], s["table"])
    return s["handle"].layer(s["q"], s["k"], s["v"], causal=s["causal"])


# --------------------------------------------------------------------------- work and tolerance
def work(case):
    kind = case["kind"]
    if kind == "gemm":
        T, N, K = case["tokens"], case["out"], case["in"]
        return {"bytes": 2.0 * (T * K + K * N + T * N), "flops": 2.0 * T * N * K}
    if kind == "linear_e4m3":
        T, N, K = case["tokens"], case["out"], case["in"]
        return {"bytes": 2.0 * T * K + 1.0 * N * K + 2.0 * T * N, "flops": 2.0 * T * N * K}
    if kind == "tp_mlp":
        T, D, F = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2.0 * (2 * T * D + T * F + 2 * D * F), "flops": 4.0 * T * D * F}
    if kind == "tp_mlp_train":
        # forward 2 products, backward 4; x, dy, w1, w2 in, y, dx, dw1, dw2 out
        T, D, F = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2.0 * (4 * T * D + 4 * D * F), "flops": 12.0 * T * D * F}
    if kind == "moe":
        T, D, F, E, K = (case[k] for k in ("tokens", "hidden", "ffn", "experts", "top_k"))
        used = E * (1.0 - (1.0 - K / E) ** T)            # experts that some token goes to, for an even router
        return {"bytes": (1.0 if case["e4m3"] else 2.0) * used * 3 * D * F + 4.0 * T * D + 4.0 * T * E, "flops": 6.0 * T * K * D * F}
    if kind == "decode":
        tokens = case["batch"] * 0.5 * (case["length"] + case["shortest"])
        return {"bytes": 4.0 * tokens * case["kv_heads"] * HEAD_DIM + 4.0 * case["batch"] * case["q_heads"] * HEAD_DIM,
                "flops": 4.0 * tokens * case["q_heads"] * HEAD_DIM}
    T, Hq, Hkv = case["tokens"], case["q_heads"], case["kv_heads"]
    return {"bytes": 4.0 * T * (Hq + Hkv) * HEAD_DIM, "flops": 4.0 * T * T * Hq * HEAD_DIM * (0.5 if case["causal"] else 1.0)}


def tolerance(case):
    # about four times the distance (2-norm) of the outputs from a 32- or 64-bit evaluation of the same inputs:
    # measured 1.7e-3 to 3.4e-3 with bf16 values, 2.1e-4 to 4.3e-4 with fp16 ones, and 1.7e-2 for the e4m3 MoE, whose
    # hidden activations are rounded to 4 significant bits (a different order of sums moves some of them by a whole step)
    if case["kind"] == "moe" and case["e4m3"]:
        return {"rel": 3e-2}
    return {"rel": 2e-3 if case.get("dtype") == "fp16" else 1e-2}
