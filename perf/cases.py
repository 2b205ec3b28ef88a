"""The work this framework is timed on: the public entry points of the W8A8 multi-LoRA path over their real range.

A case is a dict of plain values.  `op` names the entry point:

  linear       ops.w8a8_lora_linear on packed weights and tables
  grouped      ops.w8a8_lora_linear on the reference's own storage: one scale per `group` values of K, W8 or W4
  qkv          projections.FusedLoRALinearW8: one projection over [batch, tokens, K], split into q, k and v
  gate_up      ops.w8a8_rms_gate_up_lora_swiglu
  down         ops.w8a8_down_lora_residual
  block        mlp.Qwen3_5MLP.forward_with_post_attention_rms: the whole MLP block of one layer
  decode_step  stack.MLPStack over `layers` blocks, replayed from one CUDA graph as a serving loop does
  train        backward.w8a8_lora_linear_trainable: forward, backward, and the SGD step of the adapters
               (which is why a training program meets new LoRA tables on every pass)

`ids` says how token rows pick their adapter: "uniform" (every row draws one), "runs" (contiguous runs of 512 rows,
as prompts packed one after the other), "sequence" (one id per sequence), "none" (one adapter, no ids).
"""

from __future__ import annotations

import math

import torch

import skyrl_tx_rocm_b200 as S
from skyrl_tx_rocm_b200 import backward, mlp, projections, stack
from skyrl_tx_rocm_b200.weights import PackedMLPWeights

# (hidden, intermediate) of the MLPs: the Qwen3-8B and Qwen3-32B shapes of the benchmark, and generic ones
MLP_SHAPES = ((1024, 3072), (2048, 6144), (2560, 9728), (4096, 12288), (5120, 13824), (5120, 25600))


def listed():
    return [
        # a single projection of a small model: four short kernels, bound by launches and by the host
        {"name": "linear_256", "op": "linear", "m": 256, "k": 1024, "n": 3072, "rank": 8, "adapters": 1, "ids": "none"},
        # one request decoding alone: the smallest call of the block, latency of the chain and the host path
        {"name": "block_1", "op": "block", "m": 1, "hidden": 4096, "inter": 12288, "rank": 16, "adapters": 32, "ids": "uniform"},
        # a full decode batch of a serving replica with many tenants: more rows than one tile, almost every row its
        # own neighbour's stranger
        {"name": "block_256_tenants", "op": "block", "m": 256, "hidden": 4096, "inter": 12288, "rank": 16, "adapters": 32, "ids": "uniform"},
        # one chunk of chunked prefill mixed with decodes: ragged rows, a few adapters
        {"name": "block_777", "op": "block", "m": 777, "hidden": 4096, "inter": 12288, "rank": 8, "adapters": 5, "ids": "uniform"},
        # one decode step of all 36 layers of the Qwen3-8B-shaped model, 64 requests over 32 adapters
        {"name": "decode_step_64", "op": "decode_step", "m": 64, "hidden": 4096, "inter": 12288, "rank": 16, "adapters": 32, "ids": "uniform", "layers": 36},
        # prefill front half at the Qwen3-8B shape
        {"name": "gate_up_8192", "op": "gate_up", "m": 8192, "k": 4096, "n": 24576, "rank": 32, "adapters": 4, "ids": "runs"},
        # prefill back half at the Qwen3-8B shape
        {"name": "down_16384", "op": "down", "m": 16384, "k": 12288, "n": 4096, "rank": 32, "adapters": 8, "ids": "uniform"},
        # the largest: one layer of the Qwen3-32B-shaped stack on a full token batch
        {"name": "block_16384", "op": "block", "m": 16384, "hidden": 5120, "inter": 25600, "rank": 64, "adapters": 16, "ids": "uniform"},
        # attention's fused q/k/v projection on four prompts of 512 tokens (32 query heads, 8 key-value heads of 128)
        {"name": "qkv_4x512", "op": "qkv", "batch": 4, "tokens": 512, "k": 4096, "q_per_kv": 4, "kv_heads": 8, "head": 128, "rank": 16, "adapters": 4, "ids": "sequence"},
        # a checkpoint in the reference's native group-64 format, attention's output projection
        {"name": "grouped_512", "op": "grouped", "m": 512, "k": 4096, "n": 4096, "rank": 16, "adapters": 4, "ids": "uniform", "group": 64, "bits": 8},
        # LoRA fine-tuning of the down projection for eight tenants at once
        {"name": "train_4096", "op": "train", "m": 4096, "k": 12288, "n": 4096, "rank": 32, "adapters": 8, "ids": "uniform"},
        # LoRA fine-tuning of one adapter of a small model on a ragged batch
        {"name": "train_1000", "op": "train", "m": 1000, "k": 1024, "n": 3072, "rank": 8, "adapters": 1, "ids": "none"},
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], uniform over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(("linear", "block", "block", "decode_step", "gate_up", "down", "qkv", "grouped", "train"))
    rank = rng.choice((4, 8, 16, 32, 48, 64))
    adapters = _log_int(rng, 1, 32)
    ids = rng.choice(("uniform", "uniform", "runs")) if adapters > 1 else "none"
    hidden, inter = rng.choice(MLP_SHAPES)
    lora = {"rank": rank, "adapters": adapters, "ids": ids}
    if op == "linear":
        return {"op": op, "m": _log_int(rng, 1, 16384), "k": hidden, "n": _log_int(rng, 256, 25600), **lora}
    if op == "gate_up":
        return {"op": op, "m": _log_int(rng, 1, 16384), "k": hidden, "n": 2 * inter, **lora}
    if op == "down":
        return {"op": op, "m": _log_int(rng, 1, 16384), "k": inter, "n": hidden, **lora}
    if op == "block":
        return {"op": op, "m": _log_int(rng, 1, 16384), "hidden": hidden, "inter": inter, **lora}
    if op == "decode_step":
        most = max(2, min(36, int(5.4e9 / (3.0 * hidden * inter))))
        return {"op": op, "m": _log_int(rng, 1, 128), "hidden": hidden, "inter": inter, "layers": rng.randint(2, most),
                **lora, "rank": min(rank, 32)}
    if op == "qkv":
        return {"op": op, "batch": _log_int(rng, 1, 16), "tokens": _log_int(rng, 1, 1024), "k": hidden, "q_per_kv": rng.choice((2, 4, 8)),
                "kv_heads": rng.choice((4, 8)), "head": 128, "rank": rank, "adapters": adapters, "ids": "sequence" if adapters > 1 else "none"}
    if op == "grouped":
        return {"op": op, "m": _log_int(rng, 16, 2048), "k": rng.choice((1024, 2048, 4096)), "n": _log_int(rng, 512, 6144),
                **lora, "group": rng.choice((64, 128, 256)), "bits": rng.choice((4, 8))}
    return {"op": op, "m": _log_int(rng, 64, 8192), "k": rng.choice((hidden, inter)), "n": 32 * _log_int(rng, 16, 384), **lora}


# ---------------------------------------------------------------------------------------------- inputs
class _Make:
    """Seeded inputs on the GPU with the distributions of the benchmark's configurations."""

    def __init__(self, seed):
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.device)
        self.gen.manual_seed(seed)

    def normal(self, *shape, std=1.0):
        t = torch.randn(shape, generator=self.gen, device=self.device, dtype=torch.bfloat16)
        return t if std == 1.0 else t.mul_(std)

    def frozen(self, k, n, *, bits=8, group=None):
        return S.quantize_frozen_weight(self.normal(k, n, std=0.02), bits=bits, group_size=group)

    def weight(self, k, n):
        return S.pack_weight(self.frozen(k, n))

    def tables(self, adapters, k, n, rank):
        """LoRA A ~ N(0, 1 / sqrt(K)), B ~ N(0, 0.02), alpha / r = 2, in the reference's layout."""
        a = self.normal(adapters, k, rank, std=k ** -0.5)
        b = self.normal(adapters, rank, n, std=0.02)
        return a, b, torch.full((adapters,), 2.0, dtype=torch.float32, device=self.device)

    def lora(self, adapters, k, n, rank, weight):
        return S.pack_lora(*self.tables(adapters, k, n, rank), in_features=weight.in_features,
                           padded_out_features=weight.padded_out_features)

    def ids(self, kind, count, adapters):
        if kind == "none":
            return None
        if kind == "runs":
            runs = torch.randint(0, adapters, ((count + 511) // 512,), generator=self.gen, device=self.device, dtype=torch.int32)
            return runs.repeat_interleave(512)[:count].contiguous()
        return torch.randint(0, adapters, (count,), generator=self.gen, device=self.device, dtype=torch.int32)


def _block_parts(mk, c):
    gate_up, down = mk.weight(c["hidden"], 2 * c["inter"]), mk.weight(c["inter"], c["hidden"])
    return (mk.normal(c["hidden"], std=0.02), gate_up, mk.lora(c["adapters"], c["hidden"], 2 * c["inter"], c["rank"], gate_up),
            down, mk.lora(c["adapters"], c["inter"], c["hidden"], c["rank"], down))


def prepare(case, seed):
    c, mk = case, _Make(seed)
    s = {"op": c["op"]}
    if c["op"] in ("linear", "gate_up", "down"):
        w = mk.weight(c["k"], c["n"])
        s["weight"], s["lora"] = w, mk.lora(c["adapters"], c["k"], c["n"], c["rank"], w)
        x = mk.normal(c["m"], c["k"])
        if c["op"] == "gate_up":
            s["delta"] = mk.normal(c["k"], std=0.02)
        if c["op"] == "down":   # the input of a down projection is a SwiGLU product
            x = torch.nn.functional.silu(x) * mk.normal(c["m"], c["k"])
            s["residual"] = mk.normal(c["m"], c["n"])
        s["x"], s["ids"] = x, mk.ids(c["ids"], c["m"], c["adapters"])
    elif c["op"] == "grouped":
        s["weight"] = S.pack_weight(mk.frozen(c["k"], c["n"], bits=c["bits"], group=c["group"]))
        s["lora"] = mk.lora(c["adapters"], c["k"], c["n"], c["rank"], s["weight"])
        s["x"], s["ids"] = mk.normal(c["m"], c["k"]), mk.ids(c["ids"], c["m"], c["adapters"])
    elif c["op"] == "qkv":
        sizes = (c["q_per_kv"] * c["head"], c["head"], c["head"])
        n = c["kv_heads"] * sum(sizes)
        w = mk.weight(c["k"], n)
        s["layer"] = projections.FusedLoRALinearW8(w, mk.lora(c["adapters"], c["k"], n, c["rank"], w),
                                                   components=("q", "k", "v"), group_sizes=sizes, enabled=True)
        s["x"], s["ids"] = mk.normal(c["batch"], c["tokens"], c["k"]), mk.ids(c["ids"], c["batch"], c["adapters"])
    elif c["op"] == "block":
        delta, gate_up, gate_up_lora, down, down_lora = _block_parts(mk, c)
        config = mlp.W8A8BackendConfig(w8a8_mlp=True, max_lora_adapters=c["adapters"], max_lora_rank=c["rank"])
        s["layer"] = mlp.Qwen3_5MLP(config, PackedMLPWeights(gate_up, down), gate_up_lora, down_lora)
        s["norm"] = mlp.RMSNormWeights(delta)
        s["x"], s["ids"] = mk.normal(c["m"], c["hidden"]), mk.ids(c["ids"], c["m"], c["adapters"])
    elif c["op"] == "decode_step":
        s["stack"] = stack.MLPStack([_block_parts(mk, c) for _ in range(c["layers"])], num_chunks=1)
        s["x"], s["ids"] = mk.normal(c["m"], c["hidden"]), mk.ids(c["ids"], c["m"], c["adapters"])
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):   # workspaces and buffers exist before the capture
            s["stack"](s["x"], s["ids"])
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            s["out"] = s["stack"](s["x"], s["ids"])
    elif c["op"] == "train":
        s["weight"] = mk.weight(c["k"], c["n"])
        s["weight_bwd"] = backward.pack_weight_backward(s["weight"])
        a, b, s["scaling"] = mk.tables(c["adapters"], c["k"], c["n"], c["rank"])
        if c["ids"] == "none":      # the reference's single-adapter layout
            a, b, s["scaling"] = a[0], b[0], s["scaling"][0]
        s["a"], s["b"] = a.contiguous().requires_grad_(), b.contiguous().requires_grad_()
        s["x"], s["ids"] = mk.normal(c["m"], c["k"]).requires_grad_(), mk.ids(c["ids"], c["m"], c["adapters"])
        s["dy"] = mk.normal(c["m"], c["n"], std=1.0 / c["m"])
    else:
        raise ValueError(f"unknown op {c['op']!r}")
    return s


# ---------------------------------------------------------------------------------------------- one pass
def run(state):
    s = state
    op = s["op"]
    if op in ("linear", "grouped"):
        return S.w8a8_lora_linear(s["x"], s["weight"], s["lora"], adapter_ids=s["ids"], enabled=True)
    if op == "qkv":
        return s["layer"](s["x"], s["ids"])
    if op == "gate_up":
        return S.w8a8_rms_gate_up_lora_swiglu(s["x"], s["delta"], s["weight"], s["lora"], adapter_ids=s["ids"], enabled=True)
    if op == "down":
        return S.w8a8_down_lora_residual(s["x"], s["weight"], s["lora"], residual=s["residual"], adapter_ids=s["ids"], enabled=True)
    if op == "block":
        return s["layer"].forward_with_post_attention_rms(s["x"], s["norm"], s["ids"], residual=s["x"])
    if op == "decode_step":
        s["graph"].replay()
        return s["out"]
    y = backward.w8a8_lora_linear_trainable(s["x"], s["weight"], s["weight_bwd"], s["a"], s["b"], s["scaling"], s["ids"])
    dx, da, db = torch.autograd.grad(y, (s["x"], s["a"], s["b"]), s["dy"])
    with torch.no_grad():
        s["a"].sub_(da, alpha=1e-3)
        s["b"].sub_(db, alpha=1e-3)
    return {"y": y, "dx": dx, "da": da, "db": db, "a": s["a"], "b": s["b"]}


# ---------------------------------------------------------------------------------------------- what a pass needs
def _projection(m, k, n, rank, adapters):
    """(bytes, operations) of the operands of one projection: codes, scales, the tables of the adapters that can occur."""
    return (k * n + 4 * n + 2 * min(adapters, m) * rank * (k + n), 2.0 * m * k * n + 2.0 * m * rank * (k + n))


def work(case):
    """Every input read once and every output written once; an int8 multiply-add counts as two operations."""
    c = case
    if c["op"] == "qkv":
        m, n = c["batch"] * c["tokens"], c["kv_heads"] * (c["q_per_kv"] + 2) * c["head"]
        b, f = _projection(m, c["k"], n, c["rank"], c["adapters"])
        return {"bytes": b + 2 * m * (c["k"] + n) + 4 * c["batch"], "flops": f}
    m = c["m"]
    if c["op"] in ("block", "decode_step"):
        gb, gf = _projection(m, c["hidden"], 2 * c["inter"], c["rank"], c["adapters"])
        db, df = _projection(m, c["inter"], c["hidden"], c["rank"], c["adapters"])
        layers = c.get("layers", 1)
        return {"bytes": layers * (gb + db + 2 * c["hidden"]) + 4 * m * c["hidden"] + 4 * m, "flops": layers * (gf + df)}
    k, n, rank = c["k"], c["n"], c["rank"]
    b, f = _projection(m, k, n, rank, c["adapters"])
    if c["op"] == "gate_up":
        return {"bytes": b + 2 * m * k + 2 * k + m * n + 4 * m, "flops": f}
    if c["op"] == "down":
        return {"bytes": b + 2 * m * (k + 2 * n) + 4 * m, "flops": f}
    if c["op"] == "grouped":
        return {"bytes": b + 4 * n * (k // c["group"] - 1) + 2 * m * (k + n) + 4 * m, "flops": f}
    if c["op"] == "train":
        # forward, input gradient (the codes once per direction), dA and dB, gradients and updated tables written
        tables = 2 * c["adapters"] * rank * (k + n)
        return {"bytes": b + k * n + 2 * tables + 4 * m * (k + n) + 4 * m, "flops": 2 * f + 4.0 * m * rank * (k + n)}
    return {"bytes": b + 2 * m * (k + n) + 4 * m, "flops": f}


def tolerance(case):
    """bf16 results: one rounding of every value.  Through a block a one-step difference of the hidden activations
    may move an int8 code; over a stack of blocks such moves add up to the size of the quantisation noise itself."""
    return {"rel": 2e-2} if case["op"] == "decode_step" else {"rel": 1e-2}
