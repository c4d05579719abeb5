"""The work this framework is measured by: cases, their inputs, one pass, and what a pass needs.

A case is one of four kinds of work, each through the public entry points:

    layer    one step of ``InferenceMoE.run`` on a batch that is on the GPU.  ``graph`` replays a
             captured step, the way a serving loop runs decode and short prefill steps over its
             own static buffers; without it the step is launched call by call.
    grouped  ``lightmoe.gemm.GroupedGemm`` on operands packed beforehand (an expert-parallel host
             that owns routing and exchange calls just this).
    dense    ``quantize`` of the activations (FP32 or BF16, scale given or measured) and
             ``DenseGemm`` against packed weights: a linear layer in NVFP4.
    pack     ``quantize_grouped`` with measured scales: a batch and the experts' weights on their
             way from BF16 or FP32 to NVFP4, as at loading time.

Layer sizes are those of the repository's benchmark (``nvfp4moe_b200.bench_configs``); drawn
cases take those and generic ones around them.
"""

import math

import torch

from nvfp4moe_b200 import InferenceMoE
from nvfp4moe_b200.gemm import DenseGemm, GroupedGemm, quantize, quantize_grouped

NVFP4_BYTES = 0.5625  # half a byte of code and a sixteenth of a scale byte per element


def _layer(name, hidden, intermediate, experts, top_k, tokens, activation="swiglu", clamp=0.0, routing="uniform",
           graph=False):
    case = {"kind": "layer", "hidden": hidden, "intermediate": intermediate, "experts": experts, "top_k": top_k,
            "tokens": tokens, "activation": activation, "clamp": clamp, "routing": routing, "graph": graph}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one user generating, a large model with all experts on one GPU, replayed step
        _layer("decode_1", 6144, 2048, 256, 8, 1, graph=True),
        # the smallest call: one token on a small expert shard, launched call by call
        _layer("decode_1_small_eager", 2048, 512, 16, 8, 1),
        # a small batch of users on the large model
        _layer("decode_8", 6144, 2048, 256, 8, 8, graph=True),
        # a full decode batch, or the chunk of a prompt, on a shard of eight experts
        _layer("step_128", 4096, 2048, 8, 6, 128, "swiglu", 10.0, graph=True),
        # a prompt of odd length, the ungated activation, sizes that fill no tile evenly
        _layer("prefill_1777_relu2", 2688, 1920, 8, 6, 1777, "relu2"),
        # the headline layer: many thin experts
        _layer("prefill_8192", 2048, 512, 256, 8, 8192),
        # a shard of few experts with thousands of rows each
        _layer("prefill_8192_shard", 4096, 1024, 16, 10, 8192),
        # skewed routing, empty experts and one hot expert
        _layer("prefill_16384_zipf", 6144, 3072, 128, 4, 16384, "swiglu_oai", 0.0, "zipf"),
        # the largest batch
        _layer("prefill_32768", 4096, 2048, 256, 6, 32768, "swiglu", 10.0),
        # the grouped GEMM alone, small, two experts without rows
        {"name": "grouped_512", "kind": "grouped", "experts": 8, "rows": 512, "n": 1024, "k": 2048, "out": "bf16"},
        # a linear layer
        {"name": "dense_8192", "kind": "dense", "rows": 8192, "n": 4096, "k": 4096, "dtype": "bf16", "scaled": True,
         "out": "bf16"},
        # packing a batch and its experts' weights
        {"name": "pack_weights", "kind": "pack", "rows": 8192, "experts": 128, "n": 1024, "k": 2048, "dtype": "bf16"},
    ]


# hidden, intermediate, experts, top_k, activation, clamp, routing
_MODELS = (
    (2048, 512, 256, 8, "swiglu", 0.0, "uniform"),
    (4096, 2048, 256, 6, "swiglu", 10.0, "uniform"),
    (6144, 2048, 256, 8, "swiglu", 0.0, "uniform"),
    (6144, 3072, 128, 4, "swiglu_oai", 0.0, "zipf"),
    (2048, 512, 16, 8, "swiglu", 0.0, "uniform"),
    (4096, 1024, 16, 10, "swiglu", 0.0, "uniform"),
    (4096, 2048, 8, 6, "swiglu", 10.0, "uniform"),
    (6144, 2048, 16, 8, "swiglu", 0.0, "uniform"),
    (6144, 3072, 8, 4, "swiglu_oai", 0.0, "uniform"),
    (2688, 1920, 8, 6, "relu2", 0.0, "uniform"),
)


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    largest = _cost(listed()[8])
    while True:
        case = _draw(rng)
        if _cost(case) <= largest:
            return case


def _draw(rng):
    kind = rng.choices(("layer", "grouped", "dense", "pack"), (70, 10, 12, 8))[0]
    if kind == "layer":
        hidden, inter, experts, top_k, act, clamp, routing = rng.choice(_MODELS)
        if rng.random() < 0.4:
            # a model the benchmark does not have
            hidden, inter = 128 * rng.randint(8, 56), 128 * rng.randint(2, 28)
            experts = _log_int(rng, 4, 256)
            top_k = rng.randint(1, min(10, experts))
            act = rng.choice(("swiglu", "swiglu_oai", "geglu", "reglu", "relu2"))
            clamp = 10.0 if act == "swiglu" and rng.random() < 0.5 else 0.0
            routing = rng.choice(("uniform", "zipf"))
        tokens = _log_int(rng, 1, 96) if rng.random() < 0.45 else _log_int(rng, 97, 32768)
        return _layer(None, hidden, inter, experts, top_k, tokens, act, clamp, routing,
                      graph=tokens <= 512 and rng.random() < 0.5)
    n, k = 128 * rng.randint(4, 48), 64 * rng.randint(8, 96)
    if kind == "grouped":
        return {"kind": "grouped", "experts": _log_int(rng, 2, 128), "rows": _log_int(rng, 64, 65536), "n": n, "k": k,
                "out": rng.choice(("bf16", "bf16", "fp32"))}
    if kind == "dense":
        return {"kind": "dense", "rows": _log_int(rng, 16, 32768), "n": n, "k": k, "dtype": rng.choice(("bf16", "fp32")),
                "scaled": rng.random() < 0.5, "out": rng.choice(("bf16", "fp32"))}
    return {"kind": "pack", "rows": _log_int(rng, 64, 16384), "experts": _log_int(rng, 2, 128), "n": n, "k": k,
            "dtype": rng.choice(("bf16", "fp32"))}


def _cost(case):
    """What a pass takes at about 5 TB/s and 4 PFLOP/s, intermediate rows included."""
    w = work(case)
    extra = 6.0 * case["tokens"] * case["top_k"] * case["hidden"] if case["kind"] == "layer" else 0.0
    return (w["bytes"] + extra) / 5e12 + w["flops"] / 4e15


# ------------------------------------------------------------------ inputs
_FLOATS = {"bf16": torch.bfloat16, "fp32": torch.float32}


def _normal(g, *shape, std=1.0, dtype=torch.bfloat16):
    t = torch.randn(*shape, generator=g, device="cuda", dtype=dtype)
    return t.mul_(std) if std != 1.0 else t


def _routes(g, tokens, experts, top_k, routing):
    """Expert ids and renormalised weights of every token: softmax of N(0, 1) logits, or experts
    whose popularity falls as rank ** -1.2 and whose least popular sixth gets nothing."""
    if routing == "zipf":
        order = torch.randperm(experts, generator=g, device="cuda")
        popularity = torch.empty(experts, device="cuda")
        popularity[order] = torch.arange(1, experts + 1, device="cuda", dtype=torch.float32) ** -1.2
        used = max(top_k, experts - experts * 20 // 128)
        popularity[order[used:]] = 0.0
        keys = -torch.log(torch.rand(tokens, experts, generator=g, device="cuda")) / popularity
        ids = keys.topk(top_k, dim=1, largest=False).indices
        weights = torch.rand(tokens, top_k, generator=g, device="cuda") + 0.1
    else:
        logits = torch.randn(tokens, experts, generator=g, device="cuda")
        weights, ids = torch.topk(torch.softmax(logits, -1), top_k, dim=-1)
    weights = weights / weights.sum(-1, keepdim=True)
    return ids.to(torch.int32).contiguous(), weights.float().contiguous()


def _bounds(g, rows, experts):
    """Row bounds of the experts: every row picks one, two experts in eight get none."""
    picks = torch.randint(0, experts, (rows,), generator=g, device="cuda")
    if experts >= 8:
        picks = torch.where(picks % 8 == 3, picks - 1, torch.where(picks % 8 == 6, picks - 1, picks))
    bounds = torch.zeros(experts + 1, dtype=torch.int32, device="cuda")
    bounds[1:] = torch.bincount(picks, minlength=experts).cumsum(0)
    return bounds


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return {"layer": _prepare_layer, "grouped": _prepare_grouped, "dense": _prepare_dense,
            "pack": _prepare_pack}[case["kind"]](case, g)


def _prepare_layer(case, g):
    hidden, inter, experts, top_k, tokens = (case[n] for n in ("hidden", "intermediate", "experts", "top_k", "tokens"))
    layer = InferenceMoE(hidden, inter, experts, top_k, tokens, activation=case["activation"],
                         activation_clamp=case["clamp"] or None)
    first = [_normal(g, experts, inter, hidden, std=0.02) for _ in range(1 if case["activation"] == "relu2" else 2)]
    layer.load_weights(*first, _normal(g, experts, hidden, inter, std=0.02))
    x = _normal(g, tokens, hidden)
    ids, weights = _routes(g, tokens, experts, top_k, case["routing"])
    layer.calibrate(x, ids, weights)
    state = {"kind": "layer", "layer": layer, "x": x, "ids": ids, "weights": weights, "graph": None}
    if case["graph"]:
        layer.warmup(x, ids, weights)
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"]):
            layer.run(x, ids, weights)
    return state


def _tiles(rows_per_group, n):
    """The tile a caller asks for: tall on CTA pairs once a group has rows for it."""
    return (256 if rows_per_group >= 512 and n % 256 == 0 else 128), (256 if n % 256 == 0 else 128)


def _prepare_grouped(case, g):
    experts, rows, n, k = case["experts"], case["rows"], case["n"], case["k"]
    bounds = _bounds(g, rows, experts)
    operands = quantize_grouped(_normal(g, rows, k), _normal(g, experts, n, k, std=0.02), bounds)
    dtype = _FLOATS[case["out"]]
    gemm = GroupedGemm(experts, n, k, *_tiles(rows / experts, n), output_dtype=dtype)
    return {"kind": "grouped", "gemm": gemm, "operands": operands, "bounds": bounds,
            "out": torch.empty(rows, n, dtype=dtype, device="cuda")}


def _prepare_dense(case, g):
    rows, n, k = case["rows"], case["n"], case["k"]
    x = _normal(g, rows, k, dtype=_FLOATS[case["dtype"]])
    qb, sfb, b_scale = quantize(_normal(g, n, k, std=0.02))
    dtype = _FLOATS[case["out"]]
    return {"kind": "dense", "gemm": DenseGemm(n, k, *_tiles(rows, n), output_dtype=dtype), "x": x, "qb": qb, "sfb": sfb,
            "b_scale": b_scale, "scale": quantize(x)[2] if case["scaled"] else None,
            "out": torch.empty(rows, n, dtype=dtype, device="cuda")}


def _prepare_pack(case, g):
    rows, experts, n, k, dtype = case["rows"], case["experts"], case["n"], case["k"], _FLOATS[case["dtype"]]
    return {"kind": "pack", "a": _normal(g, rows, k, dtype=dtype), "b": _normal(g, experts, n, k, std=0.02, dtype=dtype),
            "bounds": _bounds(g, rows, experts)}


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "layer":
        layer = state["layer"]
        if state["graph"] is not None:
            state["graph"].replay()
            return layer.output[: state["x"].shape[0]]
        return layer.run(state["x"], state["ids"], state["weights"])
    if kind == "grouped":
        qa, qb, sfa, sfb, alpha = state["operands"]
        state["gemm"](qa, qb, state["out"], state["bounds"], sfa, sfb, alpha)
        return state["out"]
    if kind == "dense":
        qa, sfa, scale = quantize(state["x"], state["scale"])
        state["gemm"](qa, state["qb"], state["out"], sfa, state["sfb"], scale * state["b_scale"])
        return state["out"]
    qa, qb, sfa, sfb, alpha = quantize_grouped(state["a"], state["b"], state["bounds"])
    return {"qa": qa.view(torch.uint8), "qb": qb.view(torch.uint8), "sfa": sfa.view(torch.uint8),
            "sfb": sfb.view(torch.uint8), "alpha": alpha}


# ------------------------------------------------------------------ what a pass needs
def _touched_experts(case):
    """Experts that at least one route of the batch names, on average."""
    experts, top_k, tokens = case["experts"], case["top_k"], case["tokens"]
    if case["routing"] == "uniform":
        return experts * (1.0 - (1.0 - top_k / experts) ** tokens)
    used = max(top_k, experts - experts * 20 // 128)
    popularity = [(r + 1) ** -1.2 for r in range(used)]
    total = sum(popularity)
    return sum(1.0 - (1.0 - min(1.0, top_k * p / total)) ** tokens for p in popularity)


def work(case):
    kind = case["kind"]
    if kind == "layer":
        hidden, inter, top_k, tokens = (case[n] for n in ("hidden", "intermediate", "top_k", "tokens"))
        weights = (2 if case["activation"] == "relu2" else 3) * hidden * inter  # of one expert
        return {"bytes": _touched_experts(case) * weights * NVFP4_BYTES + tokens * (4.0 * hidden + 8.0 * top_k),
                "flops": 2.0 * tokens * top_k * weights}
    n, k, rows = case["n"], case["k"], case["rows"]
    if kind == "grouped":
        experts, size = case["experts"], 2 if case["out"] == "bf16" else 4
        touched = experts * (0.75 if experts >= 8 else 1.0)
        return {"bytes": (rows + touched * n) * k * NVFP4_BYTES + size * float(rows) * n, "flops": 2.0 * rows * n * k}
    size = 2 if case["dtype"] == "bf16" else 4
    if kind == "dense":
        return {"bytes": float(size) * rows * k + NVFP4_BYTES * n * k + (2.0 if case["out"] == "bf16" else 4.0) * rows * n,
                "flops": 2.0 * rows * n * k}
    return {"bytes": (size + NVFP4_BYTES) * (rows + float(case["experts"]) * n) * k, "flops": 0.0}


def tolerance(case):
    """Measured against the same packed operands in 64 bits: layers 1e-5 to 2.5e-4 (a sum that
    lands on the other side of a rounding boundary moves a code of the hidden row), BF16 GEMMs 0
    (the products are short and their FP32 sums nearly exact; another order may turn a rounding),
    FP32 GEMMs 2.5e-8."""
    if case["kind"] == "pack":
        return "exact"  # codes, scale factors and the product of two scales
    if case["kind"] == "layer":
        return {"rel": 1e-3}
    return {"rel": 1e-4 if case["out"] == "bf16" else 1e-6}
