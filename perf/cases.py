"""The workloads that the library's speed is judged by, as a user's program runs them.

Four kinds of work, each through the public entry points:

  fp8_linear   a linear layer on FP8 block-scaled weights: the activation is quantized in the
               path (``dispatch.per_token_group_quant``, or fused into the RMSNorm before it,
               ``norm.rms_norm_quant_fp8``), then ``dispatch.fp8_gemm_blockwise``
  w4a16        a linear layer on int4 weights: ``dispatch.w4a16``, or with ``source`` an
               imported checkpoint layer (``int4.from_gptq`` / ``int4.from_awq``)
  moe_fp8      a mixture-of-experts layer on FP8 weights: ``moe.gate_softmax_topk`` and
               ``parallel.expert_parallel_moe`` (one rank)
  moe_16       the same layer on unquantized f16 / bf16 weights, from the single steps

A case is a dict of plain values; ``prepare`` makes what a program holds before the call,
``run`` is one pass.
"""
import math

import torch

from kernel_set_b200 import activation, dispatch, int4, moe, norm, parallel

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16}


def listed():
    return [
        # One token through an attention projection of a small model: the smallest call, where
        # the launch and the host's path to it weigh as much as the 8 MB of weight.
        {"name": "w4a16_m1_4096x4096", "kind": "w4a16", "m": 1, "k": 4096, "n": 4096, "group": 128, "zeros": "eight",
         "dtype": "bf16", "source": "packed"},
        # A batch of 8 decoding streams through the fused gate/up projection of an MLP.
        {"name": "w4a16_m8_4096x28672", "kind": "w4a16", "m": 8, "k": 4096, "n": 28672, "group": 128, "zeros": "eight",
         "dtype": "bf16", "source": "packed"},
        # 32 streams through the down projection, from a GPTQ checkpoint quantized in activation
        # order: the activation's columns are gathered first, the zero-points are per column.
        {"name": "gptq_act_order_m32_14336x4096", "kind": "w4a16", "m": 32, "k": 14336, "n": 4096, "group": 128,
         "zeros": "random", "dtype": "f16", "source": "gptq_act_order"},
        # A ragged batch through a layer of an AWQ checkpoint with groups of 64.
        {"name": "awq_group64_m100_4096x11008", "kind": "w4a16", "m": 100, "k": 4096, "n": 11008, "group": 64,
         "zeros": "random", "dtype": "f16", "source": "awq"},
        # The prompt of one request (2048 tokens) through the gate/up projection.
        {"name": "w4a16_m2048_4096x28672", "kind": "w4a16", "m": 2048, "k": 4096, "n": 28672, "group": 128,
         "zeros": "eight", "dtype": "bf16", "source": "packed"},
        # Decode of 16 streams on FP8 weights: the weight is read once for 16 rows.
        {"name": "fp8_m16_7168x7168", "kind": "fp8_linear", "m": 16, "k": 7168, "n": 7168, "layout": "nk", "norm": False,
         "dtype": "bf16", "out": "bf16"},
        # A chunk of ragged size, weight stored [K,N] as the C ABI takes it, f16 in and out.
        {"name": "fp8_m2500_4096x2000_kn", "kind": "fp8_linear", "m": 2500, "k": 4096, "n": 2000, "layout": "kn",
         "norm": False, "dtype": "f16", "out": "f16"},
        # Prefill of 4096 tokens: the headline shape, behind the layer's RMSNorm.
        {"name": "fp8_m4096_7168x7168_norm", "kind": "fp8_linear", "m": 4096, "k": 7168, "n": 7168, "layout": "nk",
         "norm": True, "dtype": "bf16", "out": "bf16"},
        # One K-shard of a large row-parallel layer at 8 GPUs, with the fp32 partial it hands on.
        {"name": "fp8_m16384_3584x8192_f32", "kind": "fp8_linear", "m": 16384, "k": 3584, "n": 8192, "layout": "nk",
         "norm": False, "dtype": "bf16", "out": "f32"},
        # Decode step of 48 streams through an expert layer: a few rows for each expert.
        {"name": "moe_fp8_t48_e64", "kind": "moe_fp8", "tokens": 48, "hidden": 4096, "inter": 1536, "experts": 64,
         "topk": 8, "dtype": "bf16"},
        # Prefill through the large expert layer, 128 rows for an expert on average.
        {"name": "moe_fp8_t4096_e256", "kind": "moe_fp8", "tokens": 4096, "hidden": 7168, "inter": 2048, "experts": 256,
         "topk": 8, "dtype": "bf16"},
        # A layer of few, wide experts on unquantized weights.
        {"name": "moe_bf16_t512_e8", "kind": "moe_16", "tokens": 512, "hidden": 4096, "inter": 14336, "experts": 8,
         "topk": 2, "dtype": "bf16"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["fp8_linear", "fp8_linear", "fp8_linear", "w4a16", "w4a16", "w4a16", "moe_fp8", "moe_16"])
    if kind == "fp8_linear":
        ragged = rng.random() < 0.15   # K that is no multiple of the scale block
        k = 16 * _log_int(rng, 64, 1152) if ragged else 128 * _log_int(rng, 8, 144)
        n = 16 * _log_int(rng, 32, 1024)
        m = min(_log_int(rng, 1, 16384), 16384 * 8192 * 3584 // (n * k))
        return {"kind": kind, "m": m, "k": k, "n": n, "layout": rng.choice(["nk", "kn"]),
                "norm": k % 128 == 0 and rng.random() < 0.3, "dtype": rng.choice(["bf16", "bf16", "f16"]),
                "out": rng.choice(["bf16", "bf16", "f16", "f32"])}
    if kind == "w4a16":
        k = 128 * _log_int(rng, 8, 112)
        n = 16 * _log_int(rng, 64, 1792)
        m = min(_log_int(rng, 1, 4096), 2048 * 4096 * 28672 // (n * k))
        source = rng.choice(["packed", "packed", "awq", "gptq", "gptq_act_order"])
        return {"kind": kind, "m": m, "k": k, "n": n, "group": rng.choice([128, 128, 128, 64, 32]),
                "zeros": rng.choice(["eight", "random"]), "dtype": rng.choice(["bf16", "f16"]), "source": source}
    experts = 2 ** rng.randint(3, 7)
    topk = rng.choice([2, 4, 6, 8])
    if kind == "moe_fp8":
        hidden, inter = 128 * _log_int(rng, 8, 56), 128 * _log_int(rng, 4, 24)
        return {"kind": kind, "tokens": _log_int(rng, 1, 4096), "hidden": hidden, "inter": inter, "experts": experts,
                "topk": topk, "dtype": "bf16"}
    hidden, inter = 64 * _log_int(rng, 16, 64), 64 * _log_int(rng, 8, 48)
    return {"kind": kind, "tokens": _log_int(rng, 1, 2048), "hidden": hidden, "inter": inter, "experts": experts,
            "topk": topk, "dtype": rng.choice(["bf16", "f16"])}


def _block_quantized(rows, cols, g):
    """An e4m3 weight [rows, cols] with N(0, 0.02) values and its 128 x 128 block scales."""
    w = torch.randn(-(-rows // 128) * 128, -(-cols // 128) * 128, generator=g, device="cuda").mul_(0.02)
    w[rows:], w[:, cols:] = 0, 0
    blocks = w.view(w.shape[0] // 128, 128, w.shape[1] // 128, 128)
    scale = (blocks.abs().amax(dim=(1, 3)) / 448.0).clamp_min(1e-12)
    q = (blocks / scale[:, None, :, None]).to(torch.float8_e4m3fn).view(w.shape)
    return q.view(torch.uint8)[:rows, :cols].contiguous().view(torch.float8_e4m3fn), scale


def _prepare_fp8_linear(case, g):
    m, k, n = case["m"], case["k"], case["n"]
    w, w_scale = _block_quantized(n, k, g)
    if case["layout"] == "kn":
        w, w_scale = w.view(torch.uint8).t().contiguous().view(torch.float8_e4m3fn), w_scale.t().contiguous()
    dtype = DTYPES[case["dtype"]]
    state = {"x": torch.randn(m, k, generator=g, device="cuda").to(dtype), "w": w, "w_scale": w_scale,
             "layout": case["layout"], "out": DTYPES.get(case["out"], torch.float32), "gamma": None}
    if case["norm"]:
        state["gamma"] = torch.randn(k, generator=g, device="cuda").mul_(0.1).add_(1).to(dtype)
    return state


def _run_fp8_linear(s):
    x = s["x"]
    if s["gamma"] is not None:
        x8 = torch.empty(x.shape, dtype=torch.float8_e4m3fn, device=x.device)
        x_scale = torch.empty(x.shape[0], x.shape[1] // 128, dtype=torch.float32, device=x.device)
        norm.rms_norm_quant_fp8(x8, x_scale, x, s["gamma"])
    else:
        x8, x_scale = dispatch.per_token_group_quant(x)
    return dispatch.fp8_gemm_blockwise(x8, s["w"], x_scale, s["w_scale"], b_layout=s["layout"], out_dtype=s["out"])


def _random_words(shape, g):
    return torch.randint(-2**31, 2**31, shape, generator=g, device="cuda", dtype=torch.int64).to(torch.int32)


def _prepare_w4a16(case, g):
    m, k, n, group = case["m"], case["k"], case["n"], case["group"]
    dtype = DTYPES[case["dtype"]]
    x = torch.randn(m, k, generator=g, device="cuda").to(dtype)
    scales = torch.randn(k // group, n, generator=g, device="cuda").mul_(0.02).abs_().add_(1e-3).to(dtype)
    if case["source"] == "packed":
        codes = torch.randint(0, 256, (k // 2, n), generator=g, device="cuda", dtype=torch.uint8)
        if case["zeros"] == "eight":
            zeros = torch.full_like(scales, 8)
        else:
            zeros = torch.randint(0, 16, scales.shape, generator=g, device="cuda").to(dtype)
        return {"x": x, "codes": codes, "scales": scales, "zeros": zeros, "group": group, "layer": None}
    if case["zeros"] == "eight":   # GPTQ files store zero - 1
        word = 0x77777777 if case["source"] != "awq" else -0x77777778
        qzeros = torch.full((k // group, n // 8), word, device="cuda", dtype=torch.int32)
    else:
        qzeros = _random_words((k // group, n // 8), g)
    if case["source"] == "awq":
        layer = int4.from_awq(_random_words((k, n // 8), g), qzeros, scales)
    else:
        g_idx = torch.arange(k, device="cuda", dtype=torch.int32) // group
        if case["source"] == "gptq_act_order":
            g_idx = g_idx[torch.randperm(k, generator=g, device="cuda")].contiguous()
        layer = int4.from_gptq(_random_words((k // 8, n), g), qzeros, scales, g_idx=g_idx)
    return {"x": x, "layer": layer}


def _run_w4a16(s):
    if s["layer"] is not None:
        return s["layer"](s["x"])
    return dispatch.w4a16(s["x"], s["codes"], s["scales"], s["zeros"], group_size=s["group"])


def _prepare_moe(case, g):
    tokens, hidden, inter, experts = case["tokens"], case["hidden"], case["inter"], case["experts"]
    dtype = DTYPES[case["dtype"]]
    x = torch.randn(tokens, hidden, generator=g, device="cuda").to(dtype)
    logits = torch.randn(tokens, experts, generator=g, device="cuda")
    state = {"x": x, "logits": logits, "experts": experts, "topk": case["topk"], "inter": inter}
    if case["kind"] == "moe_fp8":
        w1 = torch.empty(experts, 2 * inter, hidden, dtype=torch.float8_e4m3fn, device="cuda")
        w2 = torch.empty(experts, hidden, inter, dtype=torch.float8_e4m3fn, device="cuda")
        s1 = torch.empty(experts, 2 * inter // 128, hidden // 128, device="cuda")
        s2 = torch.empty(experts, hidden // 128, inter // 128, device="cuda")
        for e in range(experts):
            w1[e], s1[e] = _block_quantized(2 * inter, hidden, g)
            w2[e], s2[e] = _block_quantized(hidden, inter, g)
        state.update(w1=w1, s1=s1, w2=w2, s2=s2)
    else:
        w1 = torch.empty(experts, hidden, 2 * inter, dtype=dtype, device="cuda")
        w2 = torch.empty(experts, inter, hidden, dtype=dtype, device="cuda")
        for e in range(experts):
            w1[e] = torch.randn(hidden, 2 * inter, generator=g, device="cuda").mul_(0.02)
            w2[e] = torch.randn(inter, hidden, generator=g, device="cuda").mul_(0.02)
        state.update(w1=w1, w2=w2)
    return state


def _route(s):
    tokens, dev = s["x"].shape[0], s["x"].device
    weights = torch.empty(tokens, s["topk"], dtype=torch.float32, device=dev)
    ids = torch.empty(tokens, s["topk"], dtype=torch.int32, device=dev)
    moe.gate_softmax_topk(weights, ids, s["logits"], tokens, s["experts"], s["topk"])
    return weights, ids


def _run_moe_fp8(s):
    weights, ids = _route(s)
    return parallel.expert_parallel_moe(s["x"], ids, weights, s["w1"], s["s1"], s["w2"], s["s2"], s["experts"])


def _run_moe_16(s):
    x, topk, experts, inter = s["x"], s["topk"], s["experts"], s["inter"]
    tokens, hidden = x.shape
    rows, dev = tokens * topk, x.device
    weights, ids = _route(s)
    order = torch.empty(rows, dtype=torch.int32, device=dev)
    offsets = torch.empty(experts + 1, dtype=torch.int32, device=dev)
    moe.compute_permutation(order, offsets, ids, tokens, experts, topk)
    xp = moe.permute(torch.empty(rows, hidden, dtype=x.dtype, device=dev), x, order, tokens, topk, hidden)
    h = dispatch.moe(xp, s["w1"], offsets, num_experts=experts, n=2 * inter, k=hidden)
    a = activation.swiglu_packed(torch.empty(rows, inter, dtype=x.dtype, device=dev), h)
    y = dispatch.moe(a, s["w2"], offsets, num_experts=experts, n=hidden, k=inter)
    return moe.unpermute(torch.empty_like(x), y, order, weights, tokens, topk, hidden)


_PREPARE = {"fp8_linear": _prepare_fp8_linear, "w4a16": _prepare_w4a16, "moe_fp8": _prepare_moe, "moe_16": _prepare_moe}
_RUN = {"fp8_linear": _run_fp8_linear, "w4a16": _run_w4a16, "moe_fp8": _run_moe_fp8, "moe_16": _run_moe_16}


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    state = _PREPARE[case["kind"]](case, g)
    state["run"] = _RUN[case["kind"]]
    return state


def run(state):
    return state["run"](state)


def work(case):
    if case["kind"] == "fp8_linear":
        m, k, n = case["m"], case["k"], case["n"]
        out = 4 if case["out"] == "f32" else 2
        return {"bytes": 2 * m * k + n * k + 4 * -(-n // 128) * -(-k // 128) + out * m * n, "flops": 2 * m * n * k}
    if case["kind"] == "w4a16":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": k * n // 2 + 4 * (k // case["group"]) * n + 2 * m * k + 2 * m * n, "flops": 2 * m * n * k}
    tokens, hidden, inter, experts, topk = (case[f] for f in ("tokens", "hidden", "inter", "experts", "topk"))
    hit = experts * (1 - (1 - topk / experts) ** tokens)   # experts that are given a token, on average
    width = 1 if case["kind"] == "moe_fp8" else 2
    return {"bytes": int(hit * 3 * hidden * inter * width) + 4 * tokens * hidden + 4 * tokens * experts,
            "flops": 6 * tokens * topk * hidden * inter}


def tolerance(case):
    """About four times what the library differs by from the same computation in 64 bits (f32
    results: from the same sums in another order). Behind an RMSNorm a value of the normalised
    row may round to its neighbour, which shows where the output keeps more digits."""
    if case["kind"] == "fp8_linear":
        if case["out"] == "f32":
            return {"rel": 5e-4 if case["norm"] else 1e-5}
        return {"rel": 7e-3, "max": 4e-2} if case["out"] == "bf16" else {"rel": 1e-3, "max": 1e-2}
    if case["kind"] == "w4a16":
        return {"rel": 7e-3, "max": 2e-2} if case["dtype"] == "bf16" else {"rel": 1e-3, "max": 2e-3}
    return {"rel": 8e-3, "max": 8e-2} if case["dtype"] == "bf16" else {"rel": 1e-3, "max": 1e-2}
