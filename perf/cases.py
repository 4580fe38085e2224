"""The work that users of this package have it do, as cases that can be timed and compared.

Two families, each through the public entry points only:

* ``linear``  floating activations -> ``quantize_rows`` -> ``int8_gemm``: a quantised linear layer;
  ``gemm``    ``int8_gemm`` on activations that are already INT8 (what the benchmark times).
* ``layer``   floating activations and router logits -> ``quantize_rows``, ``route_topk_routes``,
  ``moe_ffn``: a whole MoE feed-forward layer of a serving loop, with its workspace;
  ``moe``     ``moe_ffn`` on INT8 activations with expert ids chosen elsewhere, without a workspace.

Weights are normal values of variance 1/K quantised by ``prepare_weight``, activations are normal
values quantised by ``quantize_rows``, router logits are N(0, 1); with ``biased`` one expert's logit
is raised by 2, and with ``masked`` one token in eight is padding.
"""

import math

import torch

import grain_gemm_b200 as gg
from grain_gemm_b200.moe import MoEWorkspace

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
OUT_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}

# A drawn case stays below the work of the largest listed one.
MOST_OPS = 6.0 * 16384 * 8 * 7168 * 2048
MOST_WEIGHTS = 3 * 256 * 7168 * 2048
MOST_GEMM_OPS = 8 * 2.0 * 8192 ** 3      # at group size 256; a finer group counts 256 / group times


def _gemm(name, kind, m, n, k, group, out):
    return dict(name=name, kind=kind, m=m, n=n, k=k, group=group, out=out)


def _moe(name, kind, tokens, hidden, inter, experts, top_k, layout, out, biased, masked):
    return dict(name=name, kind=kind, tokens=tokens, hidden=hidden, inter=inter, experts=experts,
                top_k=top_k, layout=layout, out=out, biased=biased, masked=masked)


def listed():
    return [
        # One token of a decoding loop through a projection: the smallest call, latency and launches.
        _gemm("linear_m1_n4096_k4096", "linear", 1, 4096, 4096, 256, "bf16"),
        # A decoding batch against a large square weight: a read of the weights.
        _gemm("gemm_m16_n8192_k8192", "gemm", 16, 8192, 8192, 256, "bf16"),
        # A larger decoding batch, short K, finer groups, FP16.
        _gemm("linear_m128_n7168_k2048_g128", "linear", 128, 7168, 2048, 128, "fp16"),
        # A small prefill chunk with FP32 results (the benchmark's first configuration).
        _gemm("gemm_m256_n4096_k4096_fp32", "gemm", 256, 4096, 4096, 256, "fp32"),
        # Ragged sizes: an odd number of rows, K that ends within a group.
        _gemm("gemm_m509_n4096_k4000", "gemm", 509, 4096, 4000, 256, "bf16"),
        # The finest scale groups: 8 times the promotion work of G = 256.
        _gemm("gemm_m1024_n8192_k8192_g32", "gemm", 1024, 8192, 8192, 32, "bf16"),
        # The benchmark's headline: a large prefill.
        _gemm("gemm_m8192_n8192_k8192", "gemm", 8192, 8192, 8192, 256, "bf16"),
        # One token through a layer of many small experts: eight of them are touched.
        _moe("layer_t1_h2048_i768_e128", "layer", 1, 2048, 768, 128, 8, "split", "bf16", False, False),
        # Decoding with few large experts, interleaved gate/up: a read of the experts' weights.
        _moe("layer_t16_h4096_i14336_e8", "layer", 16, 4096, 14336, 8, 2, "interleaved", "bf16", True,
             False),
        # A decoding batch over many small experts, routed elsewhere.
        _moe("moe_t512_h2048_i768_e128", "moe", 512, 2048, 768, 128, 8, "split", "bf16", False, False),
        # Prefill with few large experts, one of them favoured; some tokens are padding.
        _moe("moe_t4096_h4096_i14336_e8", "moe", 4096, 4096, 14336, 8, 2, "interleaved", "bf16", True,
             True),
        # The largest: a whole layer of 256 experts on one GPU.
        _moe("layer_t16384_h7168_i2048_e256", "layer", 16384, 7168, 2048, 256, 8, "split", "bf16", False,
             False),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    if rng.random() < 0.5:
        while True:
            kind = rng.choice(("linear", "gemm"))
            m = _log_uniform(rng, 1, 8192)
            # Widths are multiples of 64, at times any number; K is a multiple of 256 for a
            # quantised row and at times any multiple of 16 for operands that come as INT8.
            n = _log_uniform(rng, 1024, 28672)
            if rng.random() < 0.75:
                n = (n + 63) // 64 * 64
            k = _log_uniform(rng, 1024, 14336)
            step = 16 if kind == "gemm" and rng.random() < 0.4 else 256
            k = (k + step - 1) // step * step
            group = rng.choice((256, 256, 256, 128, 64, 32))
            out = rng.choice(("bf16", "bf16", "bf16", "fp16", "fp32"))
            if 2.0 * m * n * k * (256 // group) <= MOST_GEMM_OPS:
                return _gemm_without_name(kind, m, n, k, group, out)
    while True:
        tokens = _log_uniform(rng, 1, 16384)
        hidden = 256 * rng.randint(4, 28)
        inter = 256 * _log_uniform(rng, 2, 56)
        experts = rng.choice((8, 16, 32, 64, 128, 256))
        top_k = rng.choice((1, 2, 4, 6, 8))
        if (3 * experts * hidden * inter <= MOST_WEIGHTS
                and 6.0 * tokens * top_k * hidden * inter <= MOST_OPS
                and tokens * top_k * max(hidden, 2 * inter) < 2 ** 31):
            case = _moe("", rng.choice(("layer", "moe")), tokens, hidden, inter, experts, top_k,
                        rng.choice(("split", "interleaved")), rng.choice(("bf16", "bf16", "fp16")),
                        rng.random() < 0.3, rng.random() < 0.3)
            del case["name"]
            return case


def _gemm_without_name(*args):
    case = _gemm("", *args)
    del case["name"]
    return case


def _normal(shape, dtype, generator, factor=1.0):
    values = torch.randn(shape, dtype=dtype, device="cuda", generator=generator)
    return values.mul_(factor) if factor != 1.0 else values


def _quantised_rows(rows, k, group, generator):
    """INT8 activations [rows, k] and their scales; k may end within a group."""
    padded = (k + 255) // 256 * 256
    q, scales = gg.quantize_rows(_normal((rows, padded), torch.bfloat16, generator), group)
    groups = (k + group - 1) // group
    return q[:, :k].contiguous(), scales[:, :groups].contiguous()


def _expert_weights(experts, n, k, group, generator):
    """Linear INT8 weights [experts, n, k] and scales [experts, k / group, n], made a few experts
    at a time."""
    q = torch.empty((experts, n, k), dtype=torch.int8, device="cuda")
    scales = torch.empty((experts, k // group, n), dtype=torch.float32, device="cuda")
    step = max(1, 2 ** 28 // (n * k))
    for first in range(0, experts, step):
        last = min(experts, first + step)
        part, part_scales = gg.prepare_weight(
            _normal((last - first, n, k), torch.bfloat16, generator, k ** -0.5), group)
        q[first:last] = part.transpose(-2, -1)
        scales[first:last] = part_scales
    return q, scales


def prepare(case, seed):
    generator = torch.Generator(device="cuda").manual_seed(seed)
    out = DTYPES[case["out"]]
    if case["kind"] in ("linear", "gemm"):
        m, n, k, group = case["m"], case["n"], case["k"], case["group"]
        padded = (k + 255) // 256 * 256
        weight, scale_b = _expert_weights(1, n, padded, group, generator)
        state = dict(kind=case["kind"], group=group, out=out, b=weight[0][:, :k].contiguous().t(),
                     scale_b=scale_b[0][:(k + group - 1) // group].contiguous())
        if case["kind"] == "linear":
            state["x"] = _normal((m, k), torch.bfloat16 if case["out"] == "fp32" else out, generator)
        else:
            state["a"], state["scale_a"] = _quantised_rows(m, k, group, generator)
        return state
    tokens, hidden, inter = case["tokens"], case["hidden"], case["inter"]
    experts, top_k = case["experts"], case["top_k"]
    w1, s1 = _expert_weights(experts, 2 * inter, hidden, 256, generator)
    w2, s2 = _expert_weights(experts, hidden, inter, 256, generator)
    # The rows are random, so a checkpoint in either gate/up order has the same values; for the
    # interleaved layout the pairs g0, u0, g1, u1, ... are simply taken to be in place.
    logits = _normal((tokens, experts), torch.float32, generator)
    if case["biased"]:
        logits[:, 0] += 2
    mask = None
    if case["masked"]:
        mask = torch.rand((tokens,), device="cuda", generator=generator) >= 0.125
    state = dict(kind=case["kind"], top_k=top_k, logits=logits,
                 ffn=dict(w_gate_up=w1.transpose(-2, -1), w_down=w2.transpose(-2, -1), scale_gate_up=s1,
                          scale_down=s2, token_mask=mask, output_dtype=out,
                          gate_up_layout=case["layout"]))
    if case["kind"] == "layer":
        state["x"] = _normal((tokens, hidden), out, generator)
        state["ffn"]["workspace"] = MoEWorkspace()
    else:
        q, scale_x = _quantised_rows(tokens, hidden, 256, generator)
        weights, ids = gg.route_topk(logits, top_k)
        state["ffn"].update(hidden_states=q, scale_x=scale_x, topk_weights=weights, topk_ids=ids)
    return state


def run(state):
    kind = state["kind"]
    if kind == "gemm":
        return gg.int8_gemm(state["a"], state["b"], state["scale_a"], state["scale_b"],
                            group_size=state["group"], output_dtype=state["out"])
    if kind == "linear":
        q, scale = gg.quantize_rows(state["x"], state["group"])
        return gg.int8_gemm(q, state["b"], scale, state["scale_b"], group_size=state["group"],
                            output_dtype=state["out"])
    if kind == "moe":
        return gg.moe_ffn(**state["ffn"])
    q, scale_x = gg.quantize_rows(state["x"])
    weights, ids, routes = gg.route_topk_routes(state["logits"], state["top_k"],
                                                token_mask=state["ffn"]["token_mask"])
    out = gg.moe_ffn(q, topk_weights=weights, topk_ids=ids, scale_x=scale_x, routes=routes,
                     **state["ffn"])
    return {"out": out, "topk_weights": weights, "topk_ids": ids}


def work(case):
    out_bytes = OUT_BYTES[case["out"]]
    if case["kind"] in ("linear", "gemm"):
        m, n, k = case["m"], case["n"], case["k"]
        groups = (k + case["group"] - 1) // case["group"]
        activations = 2 * m * k if case["kind"] == "linear" else m * k + 4 * m * groups
        return {"bytes": activations + n * k + 4 * groups * n + out_bytes * m * n,
                "flops": 2.0 * m * n * k}
    t, h, i, e, r = (case[key] for key in ("tokens", "hidden", "inter", "experts", "top_k"))
    live = t * 7 / 8 if case["masked"] else t
    touched = e * (1.0 - (1.0 - r / e) ** live)          # experts that some token is sent to
    weights = touched * 3 * h * i * (1 + 4 / 256)
    activations = t * h * (out_bytes if case["kind"] == "layer" else 1 + 4 / 256)
    routing = 4 * t * e + 12 * t * r if case["kind"] == "layer" else 12 * t * r
    return {"bytes": weights + activations + routing + out_bytes * t * h, "flops": 6.0 * live * r * h * i}


# Four times the largest differences seen between the path and the same path with its sums in
# 64 bits and the same roundings to the output type: a few outputs round the other way (one unit
# in the last place), and in the MoE layer a few requantised values do, too.
GEMM_TOLERANCE = {"bf16": {"rel": 1.5e-4, "max": 3.2e-2}, "fp16": {"rel": 4e-5, "max": 4e-3},
                  "fp32": {"rel": 1.4e-6, "max": 8e-6}}
MOE_TOLERANCE = {"bf16": {"rel": 1.2e-3, "max": 6.4e-2}, "fp16": {"rel": 5e-4, "max": 2.5e-2}}


def tolerance(case):
    table = GEMM_TOLERANCE if case["kind"] in ("linear", "gemm") else MOE_TOLERANCE
    return table[case["out"]]
