"""What a user of this framework has it do, as measurable cases: inputs, one pass through the public entry points, the work
that the pass cannot do without and how far two correct implementations may lie apart.

Five families cover the framework's public surface:

* ``linear``   activations [M, K] times a weight packed once - the call of an inference program, from one token to a long prefill,
               in every packed format, with the activation-scale modes and the fused gated activation.
* ``operands`` the reference's form of the call: A [M, K] and B [K, N] both given on every call, either as E4M3 bytes with their
               scales or in high precision (then both are quantised within the call).
* ``grouped``  the reference's grouped GEMM of unquantised experts, A [G, M, K] times B [G, K, N].
* ``moe``      a whole mixture-of-experts feed-forward layer on one GPU: routing, dispatch, the two expert GEMMs, combine.
* ``pack``     quantising and laying out a weight, what loading a model spends its time on.
"""
from __future__ import annotations

import math

import torch

from dsl_tool_b200 import MoEWeights, fp8_gemm, grouped_gemm, linear, moe_forward, pack_weight

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}
# bytes of a packed weight (or of quantised activations) per element, scales included
_PACKED = {"fp8": 1.0, "fp8_block128": 1.0 + 4.0 / (128 * 128), "nvfp4": 0.5 + 1.0 / 16, "mxfp4": 0.5 + 1.0 / 32, "bf16": 2.0}
# a calibrated global scale: the largest activation of the outlier distribution below, and of the hidden activation
_ACT_GLOBAL_SCALE = 20.0 / 2688.0
_HIDDEN_GLOBAL_SCALE = 0.01


def _linear(name, format, m, k, n, scale="dynamic", activation="none", out="bf16", dtype="bf16"):
    case = dict(family="linear", format=format, m=m, k=k, n=n, scale=scale, activation=activation, out=out, dtype=dtype)
    return dict(case, name=name) if name else case


def _operands(name, mode, given, m, k, n, dtype="bf16"):
    case = dict(family="operands", mode=mode, given=given, m=m, k=k, n=n, dtype=dtype)
    return dict(case, name=name) if name else case


def _grouped(name, groups, m, k, n, dtype="bf16"):
    case = dict(family="grouped", groups=groups, m=m, k=k, n=n, dtype=dtype)
    return dict(case, name=name) if name else case


def _moe(name, format, tokens, experts, topk, k, h, d):
    case = dict(family="moe", format=format, tokens=tokens, experts=experts, topk=topk, k=k, h=h, d=d)
    return dict(case, name=name) if name else case


def _pack(name, format, groups, n, k, layout, gate_up, dtype="bf16"):
    case = dict(family="pack", format=format, groups=groups, n=n, k=k, layout=layout, gate_up=gate_up, dtype=dtype)
    return dict(case, name=name) if name else case


def listed():
    return [
        # one sequence generating text: one token through a square projection; latency and launches are all there is
        _linear("decode_nvfp4_m1", "nvfp4", 1, 8192, 8192),
        # a small odd batch of sequences through the 70B MLP's down projection: the long K
        _linear("decode_mxfp4_m24", "mxfp4", 24, 28672, 8192),
        # a batch of sixteen through the 8B MLP's down projection with block-scaled FP8 weights, the format FP8 checkpoints ship in
        _linear("decode_fp8_block_m16", "fp8_block128", 16, 14336, 4096),
        # a chunk of prefill of a ragged length through the 8B MLP's gate/up projection, gate folded into the GEMM
        _linear("prefill_nvfp4_swiglu_m1000", "nvfp4", 1000, 4096, 28672, scale="per_token", activation="swiglu"),
        # prefill through the 8B MLP's up projection with block-scaled FP8 weights: the default workload of the benchmark
        _linear("prefill_fp8_block_m4096", "fp8_block128", 4096, 4096, 14336),
        # a long prefill through the 70B MLP's up projection: the largest dense GEMM
        _linear("prefill_mxfp4_m8192", "mxfp4", 8192, 8192, 28672),
        # the reference's own call: E4M3 bytes and scales, B [K, N], fp32 result, at the size of its plumbing check
        _operands("operands_fp8_1024", "per_tensor", "bytes", 1024, 1024, 1024),
        # the reference's grouped GEMM as its registry documents it: equal groups of bf16, B [G, K, N]
        _grouped("grouped_bf16_8x384", 8, 384, 2048, 1408),
        # one generated token for each of 64 sequences through an MoE layer: eight rows an expert, weights stream past
        _moe("moe_nvfp4_t64", "nvfp4", 64, 64, 8, 4096, 1536, 4096),
        # a ragged middle-sized batch through the layer with block-scaled FP8 weights
        _moe("moe_fp8_block_t1500", "fp8_block128", 1500, 64, 8, 4096, 1536, 4096),
        # a full prefill batch through the layer: the largest thing the framework is used for
        _moe("moe_nvfp4_t16384", "nvfp4", 16384, 64, 8, 4096, 1536, 4096),
        # loading a weight that is stored [K, N], the reference's layout
        _pack("pack_nvfp4_kn", "nvfp4", 1, 14336, 4096, "kn", False),
    ]


def _log(rng, low, high, multiple=1):
    """A whole number between low and high, spread over the logarithm, a multiple of `multiple`."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return max(-(-low // multiple), min(high // multiple, round(v / multiple))) * multiple


def draw(rng):
    family = rng.choices(("linear", "operands", "grouped", "moe", "pack"), weights=(10, 3, 2, 5, 2))[0]
    dtype = rng.choice(("bf16", "bf16", "bf16", "fp16", "fp32"))
    if family == "linear":
        format = rng.choice(("fp8", "fp8_block128", "nvfp4", "mxfp4", "bf16"))
        k = _log(rng, 1024, 28672, 128 if format == "fp8_block128" else 32)
        n = _log(rng, 1024, 28672, 16)
        m = _log(rng, 1, 128) if rng.random() < 0.5 else _log(rng, 129, 8192)
        m = max(1, min(m, int(8192.0 * 8192 * 28672 / (4 if format == "bf16" else 2 if format.startswith("fp8") else 1) / (k * n))))
        scale = rng.choice(("dynamic", "calibrated", "per_token")) if format == "nvfp4" else "dynamic"
        activation = rng.choice(("none", "none", "swiglu"))
        out = rng.choice(("bf16", "bf16", "fp32"))
        return _linear(None, format, m, k, n, scale, activation, out, "bf16" if format == "bf16" else dtype)
    if family == "operands":
        mode = rng.choice(("per_tensor", "groupwise"))
        return _operands(None, mode, rng.choice(("bytes", "values")), _log(rng, 1, 4096), _log(rng, 512, 8192, 128),
                         _log(rng, 512, 8192, 16), dtype)
    if family == "grouped":
        return _grouped(None, rng.randint(2, 32), _log(rng, 1, 1024), _log(rng, 512, 4096, 8), _log(rng, 512, 4096, 8),
                        rng.choice(("bf16", "bf16", "fp32")))
    if family == "moe":
        experts = rng.choice((8, 16, 32, 64, 128))
        return _moe(None, rng.choice(("nvfp4", "mxfp4", "fp8_block128", "fp8", "bf16")), _log(rng, 1, 8192), experts,
                    rng.choice((1, 2, 4, 6, 8)), _log(rng, 1024, 4096, 128), _log(rng, 512, 1536, 128), _log(rng, 1024, 4096, 128))
    groups = rng.choice((1, 1, 8, 64))
    return _pack(None, rng.choice(("fp8", "fp8_block128", "nvfp4", "mxfp4")), groups, _log(rng, 512, 3072 if groups > 1 else 14336, 16),
                 _log(rng, 1024, 4096, 128), rng.choice(("nk", "kn")), rng.random() < 0.3, dtype)


def _activations(gen, shape, dtype):
    """Activations as they come: N(0, 1) with one value in a thousand at 20."""
    a = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
    big = torch.rand(shape, generator=gen, device="cuda") < 1e-3
    a = torch.where(big, torch.copysign(torch.full_like(a, 20.0), a), a)
    return a.to(_DTYPES[dtype])


def _weights(gen, shape, dtype="bf16"):
    return torch.randn(shape, generator=gen, device="cuda", dtype=_DTYPES[dtype]).mul_(0.02)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    family = case["family"]
    if family == "linear":
        w = pack_weight(_weights(gen, (case["n"], case["k"])), case["format"], gate_up_interleave=case["activation"] != "none")
        options = dict(out_dtype=_DTYPES[case["out"]])
        if case["activation"] != "none":
            options["activation"] = case["activation"]
        if case["scale"] != "dynamic":
            options["act_global_scale"] = "per_token" if case["scale"] == "per_token" else torch.full((1,), _ACT_GLOBAL_SCALE, device="cuda")
        return dict(case=case, a=_activations(gen, (case["m"], case["k"]), case["dtype"]), w=w, options=options)
    if family == "operands":
        a = _activations(gen, (case["m"], case["k"]), case["dtype"])
        b = _weights(gen, (case["k"], case["n"]), case["dtype"])
        if case["given"] == "values":
            return dict(case=case, a=a, b=b, scale_a=None, scale_b=None)
        if case["mode"] == "per_tensor":
            scale_a, scale_b = float(a.abs().amax()) / 448.0, float(b.abs().amax()) / 448.0
            qa, qb = a.float() / scale_a, b.float() / scale_b
        else:   # one scale per 128 elements along K, for every row of A and every column of B
            ga, gb = a.float().reshape(case["m"], -1, 128), b.float().reshape(-1, 128, case["n"])
            scale_a = ga.abs().amax(dim=2).div_(448.0).clamp_(min=1e-12)
            scale_b = gb.abs().amax(dim=1).div_(448.0).clamp_(min=1e-12)
            qa, qb = (ga / scale_a[:, :, None]).reshape(a.shape), (gb / scale_b[:, None, :]).reshape(b.shape)
        return dict(case=case, a=qa.to(torch.float8_e4m3fn), b=qb.to(torch.float8_e4m3fn), scale_a=scale_a, scale_b=scale_b)
    if family == "grouped":
        a = _activations(gen, (case["groups"], case["m"], case["k"]), case["dtype"])
        return dict(case=case, a=a, b=_weights(gen, (case["groups"], case["k"], case["n"]), case["dtype"]))
    if family == "moe":
        x = torch.randn((case["tokens"], case["k"]), generator=gen, device="cuda", dtype=torch.bfloat16)
        logits = torch.randn((case["tokens"], case["experts"]), generator=gen, device="cuda", dtype=torch.float32)
        w = MoEWeights.pack(_weights(gen, (case["experts"], 2 * case["h"], case["k"])), _weights(gen, (case["experts"], case["d"], case["h"])),
                            case["format"], hidden_global_scale=_HIDDEN_GLOBAL_SCALE if case["format"] == "nvfp4" else None)
        return dict(case=case, x=x, logits=logits, w=w)
    shape = (case["n"], case["k"]) if case["layout"] == "nk" else (case["k"], case["n"])
    if case["groups"] > 1:
        shape = (case["groups"],) + shape
    return dict(case=case, w=_weights(gen, shape, case["dtype"]))


def run(state):
    case = state["case"]
    family = case["family"]
    if family == "linear":
        return linear(state["a"], state["w"], **state["options"])
    if family == "operands":
        return fp8_gemm(state["a"], state["b"], state["scale_a"], state["scale_b"], mode=case["mode"])
    if family == "grouped":
        return grouped_gemm(state["a"], state["b"], case["groups"])
    if family == "moe":
        return moe_forward(state["x"], state["logits"], state["w"], case["topk"], out_dtype=torch.bfloat16)
    p = pack_weight(state["w"], case["format"], layout=case["layout"], gate_up_interleave=case["gate_up"])
    return p.q, p.scale, p.global_scale


def work(case):
    family = case["family"]
    if family == "moe":
        t, e, k, h, d = (case[x] for x in ("tokens", "experts", "k", "h", "d"))
        rows = t * case["topk"]
        used = min(e, e * (1.0 - (1.0 - case["topk"] / e) ** t))        # experts that some token is routed to
        return {"bytes": used * 3 * h * k * _PACKED[case["format"]] * (1 if d == k else (2 * k + d) / (3.0 * k)) + t * k * 2 + t * e * 4 + t * d * 2,
                "flops": 2.0 * rows * h * (2 * k + d)}
    if family == "pack":
        elements = case["groups"] * case["n"] * case["k"]
        return {"bytes": elements * (_BYTES[case["dtype"]] + _PACKED[case["format"]]), "flops": 0.0}
    m, k, n, groups = case["m"], case["k"], case["n"], case.get("groups", 1)
    flops = 2.0 * groups * m * n * k
    if family == "linear":
        columns = n // 2 if case["activation"] != "none" else n
        return {"bytes": m * k * _BYTES[case["dtype"]] + n * k * _PACKED[case["format"]] + m * columns * _BYTES[case["out"]], "flops": flops}
    if family == "operands":
        size = 1 if case["given"] == "bytes" else _BYTES[case["dtype"]]
        scales = 4 * (k // 128) * (m + n) if case["given"] == "bytes" and case["mode"] == "groupwise" else 0
        return {"bytes": (m + n) * k * size + scales + m * n * 4, "flops": flops}
    size = _BYTES[case["dtype"]]
    return {"bytes": groups * ((m + n) * k + m * n) * size, "flops": flops}


def tolerance(case):
    """About four times the difference seen when the K blocks of the same problem are summed in another order (the sums of FP4 and
    FP8 products are nearly exact in fp32; those of bf16 products are not, and a gated activation amplifies them), plus, where
    the result or an intermediate is bf16 or quantised again, the roundings that such a difference flips."""
    family, wide = case["family"], case.get("format") == "bf16"
    if family == "pack":
        return "exact"              # quantised bytes and scales follow from the formats' definitions
    if family == "moe":
        return {"rel": 3.5e-3 if wide else 1.2e-3}
    if family == "grouped":
        return {"rel": 3e-4 if case["dtype"] == "bf16" else 1e-5}
    if family == "linear" and case["out"] == "bf16":
        return {"rel": 1.6e-3 if wide else 3e-4}
    if family == "linear":
        gated = case["activation"] != "none"
        return {"rel": (1.3e-4 if gated else 3e-5) if wide else (1.2e-5 if gated else 1.5e-6)}
    return {"rel": 1e-6}
