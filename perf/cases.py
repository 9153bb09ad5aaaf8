"""The work that users of this package have it do, as cases that can be timed and compared.

Two families, each through the public classes:

* ``a2a``: one ``AllToAll.dispatch`` and one ``AllToAll.combine``, as an engine with its own
  expert kernels calls them.
* ``moe``: one forward pass of ``MoELayer`` or ``MoELayerFP8``.

Keys of a case:

  family          "a2a" or "moe"
  shape           one of SHAPES (experts, top-k, hidden, expert FFN width)
  dtype           a2a: payload, "fp8" (e4m3 and one fp32 scale per 128 columns) or "bf16"
                  moe: "bf16", "fp8" (fp32 scales) or "fp8pow2" (power-of-two scales)
  out             a2a: dtype of the combined tokens, "bf16" or "fp16"
  tokens          tokens of the pass
  max_tokens      tokens the object and the tensors are sized for; above ``tokens``, the
                  device-side ``bound_m`` says how many are valid (padded decode batches)
  zipf            exponent of the expert popularity, 0 for uniform routing
  split           a2a: send and receive halves as calls of their own (overlap with compute)
  fused           moe: the four-kernel fused path, or the plain composition
  graph           the pass is the replay of a CUDA graph that was captured once
"""

from __future__ import annotations

import math
import random

import torch

from pplx_kernels_b200 import AllToAll
from pplx_kernels_b200.models.configs import (
    DEEPSEEK_V2_LITE,
    DEEPSEEK_V3,
    MIXTRAL_8X7B,
    QWEN3_30B_A3B,
    MoEModelConfig,
)
from pplx_kernels_b200.models.moe import MoELayer, MoELayerFP8

SHAPES = {
    "deepseek-v3": DEEPSEEK_V3,
    "deepseek-v2-lite": DEEPSEEK_V2_LITE,
    "mixtral-8x7b": MIXTRAL_8X7B,
    "qwen3-30b-a3b": QWEN3_30B_A3B,
    # One GPU's share of DeepSeek-V3 on eight: 32 experts that see the rows of 256.
    "deepseek-v3-share": MoEModelConfig("deepseek-v3-share", 32, 8, 7168, 2048),
}
BLOCK = 128  # columns per fp8 scale


def _a2a(name, shape, dtype, tokens, max_tokens=0, out="bf16", zipf=0.0, split=False, graph=False):
    return {"name": name, "family": "a2a", "shape": shape, "dtype": dtype, "tokens": tokens,
            "max_tokens": max_tokens or tokens, "out": out, "zipf": zipf, "split": split,
            "graph": graph}


def _moe(name, shape, dtype, tokens, max_tokens=0, zipf=0.0, fused=False, graph=False):
    return {"name": name, "family": "moe", "shape": shape, "dtype": dtype, "tokens": tokens,
            "max_tokens": max_tokens or tokens, "zipf": zipf, "fused": fused, "graph": graph}


def listed() -> list[dict]:
    return [
        # Decode of a single sequence, calls issued one by one: the latency of the two calls.
        _a2a("a2a-v3-fp8-1", "deepseek-v3", "fp8", 1),
        # The batch that the package's headline benchmark quotes.
        _a2a("a2a-v3-fp8-128", "deepseek-v3", "fp8", 128),
        # Prefill: the largest token count of the published sweeps.
        _a2a("a2a-v3-fp8-4096", "deepseek-v3", "fp8", 4096),
        # Unquantised payload in a padded batch of odd size, send and receive halves as separate
        # calls, half-precision result.
        _a2a("a2a-v2lite-bf16-301-split", "deepseek-v2-lite", "bf16", 301, 384, out="fp16",
             split=True),
        # fp8 decode of a single sequence through the whole layer.
        _moe("moe-qwen3-fp8-1", "qwen3-30b-a3b", "fp8", 1),
        # fp8 decode of a padded batch, replayed from a CUDA graph as serving engines do.
        _moe("moe-qwen3-fp8-61-graph", "qwen3-30b-a3b", "fp8", 61, 256, graph=True),
        # bf16 decode of a small batch, calls issued one by one.
        _moe("moe-qwen3-bf16-16", "qwen3-30b-a3b", "bf16", 16, fused=True),
        # Mid-sized ragged prefill chunk with skewed experts.
        _moe("moe-v2lite-fp8-1000-zipf", "deepseek-v2-lite", "fp8", 1000, zipf=1.2),
        # A full decode step of a large expert-parallel deployment, as one of its GPUs sees it.
        _moe("moe-v3share-fp8-128", "deepseek-v3-share", "fp8", 128, fused=True),
        # Few wide experts at the batch of the package's layer benchmark, and a long prefill.
        _moe("moe-mixtral-bf16-512", "mixtral-8x7b", "bf16", 512, fused=True),
        _moe("moe-mixtral-bf16-4096", "mixtral-8x7b", "bf16", 4096, fused=True),
        # The same experts in fp8 with the scales applied by the tensor cores.
        _moe("moe-mixtral-fp8pow2-2048", "mixtral-8x7b", "fp8pow2", 2048),
    ]


def draw(rng: random.Random) -> dict:
    zipf = rng.choice([0.0, 0.0, 1.2])
    if rng.random() < 0.4:
        shape, dtype = rng.choice(["deepseek-v3", "deepseek-v2-lite"]), rng.choice(["fp8", "bf16"])
        tokens = _log_uniform(rng, 1, 4096)
        max_tokens = _padded(rng, tokens)
        return {"family": "a2a", "shape": shape, "dtype": dtype, "tokens": tokens,
                "max_tokens": max_tokens, "out": rng.choice(["bf16", "bf16", "fp16"]),
                "zipf": zipf, "split": rng.random() < 0.25,
                "graph": tokens <= 256 and rng.random() < 0.5}
    shape = rng.choice(["mixtral-8x7b", "qwen3-30b-a3b", "deepseek-v2-lite", "deepseek-v3-share"])
    dtype = rng.choice(["bf16", "fp8", "fp8pow2"])
    large = shape in ("mixtral-8x7b", "deepseek-v3-share")
    tokens = _log_uniform(rng, 1, 2048 if large and dtype == "fp8" else 4096)
    # The fused fp8 path takes up to 64 experts per GPU.
    fusable = dtype == "bf16" or SHAPES[shape].num_experts <= 64
    return {"family": "moe", "shape": shape, "dtype": dtype, "tokens": tokens,
            "max_tokens": _padded(rng, tokens), "zipf": zipf,
            "fused": fusable and rng.random() < 0.5,
            "graph": tokens <= 256 and rng.random() < 0.5}


def _log_uniform(rng: random.Random, low: int, high: int) -> int:
    return min(high, int(math.exp(rng.uniform(math.log(low), math.log(high + 1)))))


def _padded(rng: random.Random, tokens: int) -> int:
    """The size of the batch's tensors: the token count itself, or the next multiple of 64."""
    return tokens if rng.random() < 0.6 else (tokens + 63) // 64 * 64


# ------------------------------------------------------------------------- inputs ----


def _routing(gen: torch.Generator, rows: int, experts: int, topk: int, zipf: float) -> torch.Tensor:
    """[rows, topk] distinct experts per token, drawn without replacement (Gumbel top-k)."""
    dev = gen.device
    logits = -zipf * torch.log(torch.arange(1, experts + 1, device=dev, dtype=torch.float32))
    u = torch.rand(rows, experts, generator=gen, device=dev).clamp_(1e-20, 1.0)
    noise = -torch.log((-torch.log(u)).clamp_(min=1e-20))
    return (logits + noise).topk(topk, dim=1).indices.to(torch.int32).view(torch.uint32)


def prepare(case: dict, seed: int) -> dict:
    cfg = SHAPES[case["shape"]]
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    rows = case["max_tokens"]
    s: dict = {"family": case["family"]}
    s["indices"] = _routing(gen, rows, cfg.num_experts, cfg.experts_per_token, case["zipf"])
    s["weights"] = torch.softmax(
        torch.randn(rows, cfg.experts_per_token, generator=gen, device=dev), dim=-1)
    s["bound_m"] = None
    if case["tokens"] < rows:
        s["bound_m"] = torch.tensor([case["tokens"]], dtype=torch.int32, device=dev).view(torch.uint32)
    x = torch.randn(rows, cfg.hidden_dim, generator=gen, device=dev)
    if case["family"] == "a2a":
        _prepare_a2a(s, case, cfg, gen, x)
    else:
        s["x"] = x.to(torch.bfloat16)
        s["out"] = torch.zeros(rows, cfg.hidden_dim, dtype=torch.bfloat16, device=dev)
        if case["dtype"] == "bf16":
            s["layer"] = MoELayer(cfg, max_num_tokens=rows, device=dev, seed=seed)
        else:
            s["layer"] = MoELayerFP8(cfg, max_num_tokens=rows, device=dev, seed=seed,
                                     pow2_scales=case["dtype"] == "fp8pow2")
        s["fused"] = case["fused"]
    s["graph"] = None
    if case["graph"]:
        _pass(s)  # the first call of a kernel is not capturable
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            _pass(s)
    return s


def _prepare_a2a(s: dict, case: dict, cfg: MoEModelConfig, gen: torch.Generator,
                 x: torch.Tensor) -> None:
    dev, rows, hidden, experts = x.device, case["max_tokens"], cfg.hidden_dim, cfg.num_experts
    s["split"] = case["split"]
    s["x_scale"] = s["expert_scale"] = None
    if case["dtype"] == "fp8":
        blocks = x.view(rows, hidden // BLOCK, BLOCK)
        s["x_scale"] = blocks.abs().amax(dim=2).clamp(min=1e-4) / 448.0
        s["x"] = (blocks / s["x_scale"].unsqueeze(2)).view(rows, hidden).to(torch.float8_e4m3fn)
        s["expert_x"] = torch.zeros(experts, rows, hidden, dtype=torch.uint8,
                                    device=dev).view(torch.float8_e4m3fn)
        s["expert_scale"] = torch.zeros(experts, rows, hidden // BLOCK, device=dev)
        # What the experts answer.  The order of an expert's rows is not specified, so all
        # rows of one expert carry the same values: the result does not depend on it.
        answer = torch.randn(experts, 1, hidden, generator=gen, device=dev).to(torch.bfloat16)
        s["expert_y"] = answer.expand(experts, rows, hidden).contiguous()
        scale_bytes = hidden // BLOCK * 4
    else:
        # Identity experts: what was dispatched is combined.
        s["x"] = x.to(torch.bfloat16)
        s["expert_x"] = torch.zeros(experts, rows, hidden, dtype=torch.bfloat16, device=dev)
        s["expert_y"] = s["expert_x"]
        scale_bytes = 0
    s["counts"] = torch.zeros(experts, dtype=torch.int32, device=dev)
    s["out"] = torch.zeros(rows, hidden, device=dev,
                           dtype=torch.float16 if case["out"] == "fp16" else torch.bfloat16)
    s["ata"] = AllToAll.intranode(rows, experts, cfg.experts_per_token, 0, 1, 1, hidden,
                                  hidden * s["x"].element_size(), scale_bytes)
    # An expert gets one row at most from one token: its place is known, so it can be compared.
    s["whole"] = case["tokens"] == 1 and case["dtype"] == "fp8"


# --------------------------------------------------------------------------- pass ----


def _pass(s: dict) -> None:
    if s["family"] == "moe":
        s["layer"](s["x"], s["indices"], s["weights"], out=s["out"], bound_m=s["bound_m"],
                   fused=s["fused"])
        return
    ata = s["ata"]
    dispatch_args = (s["counts"], s["expert_x"], s["expert_scale"], s["x"], s["x_scale"],
                     s["indices"], s["bound_m"])
    combine_args = (s["out"], s["indices"], s["weights"], s["expert_y"], s["bound_m"])
    if s["split"]:
        ata.dispatch(*dispatch_args, do_recv=False)
        ata.dispatch(*dispatch_args, do_send=False)
        ata.combine(*combine_args, do_recv=False)
        ata.combine(*combine_args, do_send=False)
    else:
        ata.dispatch(*dispatch_args)
        ata.combine(*combine_args)


def run(s: dict) -> dict:
    if s["graph"] is not None:
        s["graph"].replay()
    else:
        _pass(s)
    if s["family"] == "moe":
        return {"out": s["out"], "counts": s["layer"].counts}
    outputs = {"out": s["out"], "counts": s["counts"]}
    if s["whole"]:
        outputs["expert_x"] = s["expert_x"].view(torch.uint8)
        outputs["expert_scale"] = s["expert_scale"]
    return outputs


# ------------------------------------------------------------------ work, tolerance ----


def work(case: dict) -> dict:
    cfg = SHAPES[case["shape"]]
    m, k, hidden = case["tokens"], cfg.experts_per_token, cfg.hidden_dim
    routing_bytes = m * k * 8 + cfg.num_experts * 4  # experts and weights in, counts out
    if case["family"] == "a2a":
        row = hidden + hidden // BLOCK * 4 if case["dtype"] == "fp8" else 2 * hidden
        # Tokens in, expert rows out; expert results in, tokens out.
        return {"bytes": m * row + m * k * row + m * k * hidden * 2 + m * hidden * 2 + routing_bytes,
                "flops": 2 * m * k * hidden}
    weight = 2 if case["dtype"] == "bf16" else 1
    expert_bytes = 3 * hidden * cfg.intermediate_dim * weight
    return {"bytes": m * hidden * 4 + _experts_touched(case, cfg) * expert_bytes + routing_bytes,
            "flops": m * cfg.flops_per_token()}


def _experts_touched(case: dict, cfg: MoEModelConfig) -> float:
    """Expected number of experts that get a token (sampling with replacement when skewed)."""
    p = [1.0 / (e + 1) ** case["zipf"] for e in range(cfg.num_experts)]
    total = sum(p)
    draws = case["tokens"] * cfg.experts_per_token
    if case["zipf"] == 0.0:
        return cfg.num_experts * (1.0 - (1.0 - cfg.experts_per_token / cfg.num_experts) ** case["tokens"])
    return sum(1.0 - (1.0 - q / total) ** draws for q in p)


def tolerance(case: dict) -> dict:
    if case["family"] == "a2a":
        # fp32 sums of top-k values, rounded once: one unit in the last place of the result.
        return {"rel": 1e-3, "max": 1e-3} if case["out"] == "fp16" else {"rel": 4e-3, "max": 8e-3}
    return {"rel": 1e-2}
