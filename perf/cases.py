"""The work that is timed when a change to the kernels or to the host path is judged.

Each case is one call (or one forward + backward) that a program built on this package makes, through the
package's public entry points:

  block         moe_block_forward without gradients: a decoding step or a prefill
  block_train   moe_block_forward and the gradients of the tokens, the router and the three projections
  linear_train  moe_fused_linear and the gradients of its input and its weight
  lora_train    fast_lora (frozen dense base weights plus LoRA) and the gradients of the tokens and the adapters
  nf4_linear    moe_fused_linear_4bit without gradients, on batches from 1400 rows per expert on (smaller ones take
                another kernel, which is not timed here)

Sizes: hidden 2048, expert width 768 (gate and up together 1536), 128 experts, 8 per token are those of bench.py and
of the tests; the second geometry is a generic smaller layer.
"""
import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "transformers-qwen3-moe-fused_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from qwen3_moe_fused.functional import moe_fused_linear  # noqa: E402
from qwen3_moe_fused.kernels.fast_lora import fast_lora  # noqa: E402
from qwen3_moe_fused.moe_block import moe_block_forward  # noqa: E402
from qwen3_moe_fused.quantize.linear4bit import moe_fused_linear_4bit  # noqa: E402
from qwen3_moe_fused.quantize.nf4 import nest_absmax, quantize_nf4  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}
#             hidden, expert width, experts, experts per token
GEOMETRY = {"large": (2048, 768, 128, 8), "small": (1024, 512, 32, 4)}


def listed():
    return [
        # serving: one sequence, then a small batch of sequences, one new token each
        {"name": "decode_1", "kind": "block", "tokens": 1, "geometry": "large", "dtype": "bf16"},
        {"name": "decode_48", "kind": "block", "tokens": 48, "geometry": "large", "dtype": "bf16"},
        # serving: a prompt of an odd length; a batch of 8 prompts of 2048 tokens
        {"name": "prefill_1777", "kind": "block", "tokens": 1777, "geometry": "large", "dtype": "bf16"},
        {"name": "prefill_16384", "kind": "block", "tokens": 16384, "geometry": "large", "dtype": "bf16"},
        # full fine-tuning of a layer on a batch of packed sequences
        {"name": "block_train_8191", "kind": "block_train", "tokens": 8191, "geometry": "large", "dtype": "bf16"},
        # the projections on their own, as a model that calls them one by one does: gate and up stacked on the rows of
        # 8192 tokens; down with skewed routing and experts that get nothing; a small batch in fp16
        {"name": "linear_gate_up_65536", "kind": "linear_train", "rows": 65536, "in": 2048, "out": 1536, "experts": 128,
         "routing": "softmax", "dtype": "bf16"},
        {"name": "linear_down_zipf_65536", "kind": "linear_train", "rows": 65536, "in": 768, "out": 2048, "experts": 128,
         "routing": "zipf", "dtype": "bf16"},
        {"name": "linear_f16_5003", "kind": "linear_train", "rows": 5003, "in": 2048, "out": 768, "experts": 128,
         "routing": "random", "dtype": "f16"},
        # LoRA fine-tuning of the expert MLP: a short sequence, an ordinary batch, and a smaller layer with a high rank,
        # fp16 and skewed routing
        {"name": "lora_512", "kind": "lora_train", "tokens": 512, "geometry": "large", "rank": 16, "routing": "softmax",
         "dtype": "bf16"},
        {"name": "lora_4096", "kind": "lora_train", "tokens": 4096, "geometry": "large", "rank": 16, "routing": "softmax",
         "dtype": "bf16"},
        {"name": "lora_small_r64_3001", "kind": "lora_train", "tokens": 3001, "geometry": "small", "rank": 64,
         "routing": "zipf", "dtype": "f16"},
        # inference on 4-bit weights whose block scales are quantised as well: the rows of 32768 tokens, where every
        # weight is decoded once for the whole batch
        {"name": "nf4_linear_262144", "kind": "nf4_linear", "rows": 262144, "in": 2048, "out": 1536, "experts": 128,
         "routing": "softmax", "nested": True, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "prefill", "block_train", "linear_train", "lora_train", "lora_train", "nf4_linear"])
    geometry = rng.choice(["large", "large", "large", "small"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "f16"])
    if kind == "decode":
        return {"kind": "block", "tokens": _log_int(rng, 1, 256), "geometry": geometry, "dtype": dtype}
    if kind == "prefill":
        return {"kind": "block", "tokens": _log_int(rng, 257, 16384), "geometry": geometry, "dtype": dtype}
    if kind == "block_train":
        return {"kind": "block_train", "tokens": _log_int(rng, 256, 8192), "geometry": geometry, "dtype": dtype}
    if kind == "lora_train":
        return {"kind": "lora_train", "tokens": _log_int(rng, 128, 8192), "geometry": geometry,
                "rank": rng.choice([8, 16, 16, 32, 64]), "routing": rng.choice(["softmax", "zipf"]), "dtype": dtype}
    k_in, n_out = rng.choice([(2048, 1536), (2048, 768), (768, 2048), (1024, 512)])
    experts = 32 if k_in == 1024 else 128
    routing = rng.choice(["softmax", "random", "zipf"])
    if kind == "linear_train":
        return {"kind": "linear_train", "rows": _log_int(rng, 1024, 65536), "in": k_in, "out": n_out, "experts": experts,
                "routing": routing, "dtype": dtype}
    return {"kind": "nf4_linear", "rows": 1400 * experts + rng.randrange(650 * experts), "in": k_in, "out": n_out,
            "experts": experts, "routing": routing, "nested": rng.random() < 0.5, "dtype": dtype}


# ------------------------------------------------------------------------------------------ inputs
def _sizes(rows, experts, routing, k, gen, dev):
    """Rows of each expert (int32): top-k of N(0,1) logits, ids drawn evenly, or Zipf(1.2) over experts in random
    order with three of them left without rows."""
    if routing == "softmax":
        logits = torch.randn(-(-rows // k), experts, generator=gen, device=dev)
        ids = logits.topk(k, dim=1).indices.reshape(-1)[:rows]
    elif routing == "random":
        ids = torch.randint(experts, (rows,), generator=gen, device=dev)
    else:
        pmf = (torch.arange(experts, device=dev, dtype=torch.float64) + 1) ** -1.2
        pmf[[5, experts // 2, experts - 1]] = 0
        cdf = (pmf / pmf.sum()).cumsum(0)
        ids = torch.searchsorted(cdf, torch.rand(rows, generator=gen, device=dev, dtype=torch.float64)).clamp_max(experts - 2)
        ids = torch.randperm(experts, generator=gen, device=dev)[ids]
    return torch.bincount(ids, minlength=experts).to(torch.int32)


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    kind = case["kind"]

    def normal(*shape, scale=1.0):
        t = torch.randn(*shape, generator=gen, device=dev, dtype=dt)
        return t if scale == 1.0 else t.mul_(scale)

    if kind in ("block", "block_train"):
        H, I, E, k = GEOMETRY[case["geometry"]]
        args = [normal(1, case["tokens"], H), normal(E, H, scale=H ** -0.5), normal(E, I, H, scale=0.02),
                normal(E, I, H, scale=0.02), normal(E, H, I, scale=0.02)]
        state = {"kind": kind, "args": args, "k": k}
        if kind == "block_train":
            for t in args:
                t.requires_grad_()
            state["dout"] = normal(1, case["tokens"], H)
        return state
    if kind == "lora_train":
        H, I, E, k = GEOMETRY[case["geometry"]]
        R, rows = case["rank"], case["tokens"] * k
        m_sizes = _sizes(rows, E, case["routing"], k, gen, dev)
        x = normal(rows, H).requires_grad_()
        args, leaves = [x], [x]
        for n_out, n_in in ((I, H), (I, H), (H, I)):  # gate, up, down
            w = normal(E, n_out, n_in, scale=0.02)
            a = normal(E, R, n_in, scale=n_in ** -0.5).requires_grad_()
            b = normal(E, n_out, R, scale=0.01).requires_grad_()
            args += [w, None, a, b, 2.0]
            leaves += [a, b]
        return {"kind": kind, "args": args + [m_sizes], "leaves": leaves, "dy": normal(rows, H)}
    rows, K, N, E = case["rows"], case["in"], case["out"], case["experts"]
    m_sizes = _sizes(rows, E, case["routing"], 8, gen, dev)
    w = normal(E, N, K, scale=0.02)
    if kind == "linear_train":
        return {"kind": kind, "x": normal(rows, K).requires_grad_(), "w": w.requires_grad_(), "m_sizes": m_sizes,
                "dy": normal(rows, N)}
    packed, state = quantize_nf4(w, 64)
    return {"kind": kind, "x": normal(rows, K), "packed": packed, "state": nest_absmax(state) if case["nested"] else state,
            "m_sizes": m_sizes}


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "block":
        with torch.no_grad():
            return moe_block_forward(*state["args"], state["k"], True)
    if kind == "block_train":
        out, logits = moe_block_forward(*state["args"], state["k"], True)
        return (out.detach(), logits.detach(), *torch.autograd.grad(out, state["args"], state["dout"]))
    if kind == "linear_train":
        y = moe_fused_linear(state["x"], state["w"], state["m_sizes"])
        return (y.detach(), *torch.autograd.grad(y, (state["x"], state["w"]), state["dy"]))
    if kind == "lora_train":
        y = fast_lora(*state["args"])
        return (y.detach(), *torch.autograd.grad(y, state["leaves"], state["dy"]))
    with torch.no_grad():
        return moe_fused_linear_4bit(state["x"], state["packed"], state["state"], state["m_sizes"])


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("block", "block_train"):
        H, I, E, k = GEOMETRY[case["geometry"]]
        T = case["tokens"]
        used = E * (1.0 - (1.0 - k / E) ** T)  # experts that get a token
        weights = 2.0 * (3 * used * H * I + E * H)
        tokens = 2.0 * T * (2 * H + E)
        flops = 2.0 * T * (k * 3 * H * I + E * H)
        if kind == "block":
            return {"bytes": weights + tokens, "flops": flops}
        return {"bytes": weights + 2.0 * (3 * E * H * I + E * H) + tokens + 2.0 * T * 2 * H, "flops": 3 * flops}
    if kind == "lora_train":
        H, I, E, k = GEOMETRY[case["geometry"]]
        R, M = case["rank"], case["tokens"] * k
        base = 3.0 * E * H * I * 2.0
        adapters = 2.0 * 3 * E * R * (H + I)
        return {"bytes": base + 2 * adapters + 2.0 * M * 4 * H, "flops": 2.0 * M * (2 * 3 * H * I + 3 * 3 * R * (H + I))}
    M, K, N, E = case["rows"], case["in"], case["out"], case["experts"]
    used = E * (1.0 - (1.0 - 1.0 / E) ** M)
    if kind == "linear_train":
        return {"bytes": 2.0 * (used * K * N + E * K * N + M * (2 * K + 2 * N)), "flops": 3 * 2.0 * M * K * N}
    scale = 1 / 64 * (1 + 4 / 256) if case["nested"] else 4 / 64
    return {"bytes": used * K * N * (0.5 + scale) + 2.0 * M * (K + N), "flops": 2.0 * M * K * N}


def tolerance(case):
    """Four times what the results differ by from the same computation in fp32 (2-norm over 2-norm 0.0017 / 0.0021 for one
    GEMM in bf16 with a dense / a decoded weight, 0.0053 to 0.0062 for the chains of three projections with the stored
    intermediates between them, an eighth of that in fp16), the chains a little less."""
    chain = case["kind"] in ("block", "block_train", "lora_train")
    rel, most = (2e-2, 0.2) if chain else (8e-3, 4e-2)
    return {"rel": rel, "max": most} if case["dtype"] == "bf16" else {"rel": rel / 8, "max": most / 8}
