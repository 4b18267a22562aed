"""The work this library is measured on: its public entry points over the range of sizes they are used at.

A case is a dict of plain values; `op` says which entry point it goes through:

    gemm      Nvfp4Gemm.run       packed operands -> C (NVFP4, or MXFP4 with format "mx")
    linear    Nvfp4Gemm.linear    16/32-bit activations -> quantised into the plan -> C
    mx_linear quantize_mx + run   the same layer in MXFP4: the activations are quantised, then multiplied
    quantize  quantize            a tensor -> packed codes + scale bytes (format "nvfp4", "scaled" = two-level, "mx")
    moe       Nvfp4MoE.forward    the routed expert layer, called as it is or replayed from its captured graph

`prepare` makes what a program holds before the call (weights quantised once, plans, layers, input tensors), `run` is
one call.
"""
import math

import torch

import gpu_kernels_b200 as g
from gpu_kernels_b200.nvfp4 import scale_rows, tensor_scale_for

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def listed():
    return [
        # One tile of work: a small projection, where the call itself and the launch are the cost.
        {"name": "gemm_256", "op": "gemm", "format": "nvfp4", "m": 256, "n": 256, "k": 256, "out": "f16"},
        # A decode step of eight sequences through an 8192 x 8192 projection: the weights stream once.
        {"name": "linear_decode_8", "op": "linear", "m": 8, "n": 8192, "k": 8192, "x": "bf16", "out": "bf16"},
        # The wide decode projection of the benchmark: 128 rows of activations against 28672 x 8192 weights.
        {"name": "gemm_skinny_128", "op": "gemm", "format": "nvfp4", "m": 128, "n": 28672, "k": 8192, "out": "f16"},
        # A prefill chunk of an odd number of tokens: ragged rows, bf16 in and out.
        {"name": "linear_prefill_1000", "op": "linear", "m": 1000, "n": 8192, "k": 8192, "x": "bf16", "out": "bf16"},
        # The headline product.
        {"name": "gemm_8192", "op": "gemm", "format": "nvfp4", "m": 8192, "n": 8192, "k": 8192, "out": "f16"},
        # The large one: operands beyond the L2 cache.
        {"name": "gemm_16384", "op": "gemm", "format": "nvfp4", "m": 16384, "n": 16384, "k": 16384, "out": "f16"},
        # Activations of a large prefill, or a weight matrix at load time.
        {"name": "quantize_bf16_8192", "op": "quantize", "format": "nvfp4", "rows": 8192, "k": 8192, "x": "bf16"},
        # FP32 master weights with a per-tensor scale (two-level NVFP4), an odd row count.
        {"name": "quantize_scaled_f32", "op": "quantize", "format": "scaled", "rows": 5003, "k": 4096, "x": "f32"},
        # The same layer in MXFP4 at a middle size.
        {"name": "mx_linear_2048", "op": "mx_linear", "m": 2048, "n": 4096, "k": 2048, "x": "f16", "out": "f16"},
        # The expert layer in a decode loop: one token, replayed from its graph.
        {"name": "moe_token_1", "op": "moe", "tokens": 1, "hidden": 4096, "inter": 2048, "experts": 256, "topk": 6,
         "skew": 0.0, "graph": True},
        # A decode batch through the expert layer.
        {"name": "moe_tokens_64", "op": "moe", "tokens": 64, "hidden": 4096, "inter": 2048, "experts": 256, "topk": 6,
         "skew": 0.0, "graph": False},
        # A prefill batch through the expert layer.
        {"name": "moe_tokens_4096", "op": "moe", "tokens": 4096, "hidden": 4096, "inter": 2048, "experts": 256, "topk": 6,
         "skew": 0.0, "graph": False},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _multiple(rng, lo, hi, of):
    return _log_int(rng, lo // of, hi // of) * of


def draw(rng):
    op = rng.choice(("gemm", "linear", "mx_linear", "quantize", "moe"))
    if op == "moe":
        experts = rng.choice((8, 16, 32, 64, 128, 256))
        tokens = _log_int(rng, 1, 4096)
        return {"op": op, "tokens": tokens, "hidden": 256 * rng.randint(4, 16), "inter": 256 * rng.randint(2, 8),
                "experts": experts, "topk": rng.randint(1, 8), "skew": rng.choice((0.0, 0.5, 1.0)),
                "graph": tokens <= 256 and rng.random() < 0.5}
    if op == "quantize":
        fmt = rng.choice(("nvfp4", "nvfp4", "scaled", "mx"))
        k = _multiple(rng, 256, 28672, 128 if fmt == "mx" else 64)
        rows = _log_int(rng, 1, max(1, min(28672, (1 << 28) // k)))
        return {"op": op, "format": fmt, "rows": rows, "k": k, "x": rng.choice(("bf16", "bf16", "f16", "f32"))}
    # products: any number of rows (decode to prefill), layer widths that need not be whole tiles
    mx = op == "mx_linear" or (op == "gemm" and rng.random() < 0.25)
    k = _multiple(rng, 512, 16384, 128 if mx else 64)
    n = _multiple(rng, 512, 28672, rng.choice((8, 128, 256)))
    m = _log_int(rng, 1, max(1, min(16384, (1 << 41) // (n * k))))
    if rng.random() < 0.3:
        m = -(-m // 128) * 128
    case = {"op": op, "m": m, "n": n, "k": k, "out": rng.choice(("f16", "bf16"))}
    if op == "gemm":
        case["format"] = "mx" if mx else "nvfp4"
    else:
        case["x"] = rng.choice(("bf16", "bf16", "f16", "f32"))
    return case


def _normal(gen, rows, k, sigma, dtype):
    """N(0, sigma) drawn as bf16 (the distribution of the benchmark's activations and weights), as `dtype`."""
    x = torch.empty((rows, k), dtype=torch.bfloat16 if dtype == torch.bfloat16 else torch.float32, device="cuda")
    return x.normal_(0.0, sigma, generator=gen).to(dtype)


def _is_mx(case):
    return case["op"] == "mx_linear" or case.get("format") == "mx"


def _product_inputs(case, gen):
    """The weights [N, K] and activations [M, K] of a product before they are quantised."""
    m, n, k = case["m"], case["n"], case["k"]
    square = case["op"] == "gemm" and m == n == k                 # the benchmark's square products are N(0,1) on both sides
    b = _normal(gen, n, k, 1.0 if square else 0.02, torch.bfloat16)
    return b, _normal(gen, m, k, 1.0, torch.bfloat16 if case["op"] == "gemm" else DTYPES[case["x"]])


def _prepare_product(case, gen):
    op, m, n, k = case["op"], case["m"], case["n"], case["k"]
    mx = _is_mx(case)
    pack = g.quantize_mx if mx else g.quantize
    b, x = _product_inputs(case, gen)
    b, sfb = pack(b)
    if op == "mx_linear":
        return {"op": op, "b": b, "sfb": sfb, "x": x, "out": case["out"]}
    state = {"op": op}
    if op == "linear":
        # the plan's own A and scales: `linear` quantises into them
        a = torch.empty((m, k // 2), dtype=torch.uint8, device="cuda")
        sfa = torch.empty(scale_rows(m) * k // 16, dtype=torch.uint8, device="cuda")
        state["x"] = x
    else:
        a, sfa = pack(x)
        state["c"] = torch.empty((m, n), dtype=DTYPES[case["out"]], device="cuda")
    state["plan"] = g.Nvfp4Gemm(a, b, sfa, sfb, mx=mx)
    if case["out"] == "bf16":
        state["plan"].set_option("out_bf16", 1)
    return state


def _moe_inputs(case, gen):
    t, h, i, e, topk = (case[key] for key in ("tokens", "hidden", "inter", "experts", "topk"))
    w1 = torch.empty((e, 2 * i, h), dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=gen)
    w2 = torch.empty((e, h, i), dtype=torch.bfloat16, device="cuda").normal_(0.0, 0.02, generator=gen)
    x = _normal(gen, t, h, 1.0, torch.bfloat16)
    logits = torch.randn((t, e), generator=gen, device="cuda")
    if case["skew"]:
        logits += case["skew"] * torch.randn((1, e), generator=gen, device="cuda")     # experts of unequal popularity
    ids, weights = g.route(logits, topk)
    return w1, w2, x, ids, weights


def _prepare_moe(case, gen):
    w1, w2, x, ids, weights = _moe_inputs(case, gen)
    # a layer is sized for the largest batch it may see
    layer = g.Nvfp4MoE(w1, w2, case["experts"], case["topk"], clamp=10.0, max_tokens=256 if case["graph"] else 4096)
    del w1, w2
    state = {"op": "moe", "layer": layer, "x": x, "ids": ids, "weights": weights}
    if case["graph"]:
        state["captured"] = layer.capture(case["tokens"])
    return state


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    op = case["op"]
    if op == "moe":
        return _prepare_moe(case, gen)
    if op == "quantize":
        x = _normal(gen, case["rows"], case["k"], 1.0, DTYPES[case["x"]])
        scale = tensor_scale_for(x) if case["format"] == "scaled" else None
        return {"op": op, "format": case["format"], "x": x, "scale": scale}
    return _prepare_product(case, gen)


def run(state):
    op = state["op"]
    if op == "gemm":
        return state["plan"].run(state["c"])
    if op == "linear":
        return state["plan"].linear(state["x"])
    if op == "mx_linear":
        # a plan holds the addresses of its operands, and the quantiser returns new tensors: one plan per call
        a, sfa = g.quantize_mx(state["x"])
        plan = g.Nvfp4Gemm(a, state["b"], sfa, state["sfb"], mx=True)
        if state["out"] == "bf16":
            plan.set_option("out_bf16", 1)
        return plan.run()
    if op == "quantize":
        if state["format"] == "mx":
            return g.quantize_mx(state["x"])
        if state["format"] == "scaled":
            return g.quantize(state["x"], tensor_scale=state["scale"])
        return g.quantize(state["x"])
    if "captured" in state:
        x, ids, weights, y, graph = state["captured"]
        x.copy_(state["x"])
        ids.copy_(state["ids"])
        weights.copy_(state["weights"])
        graph.replay()
        return y
    return state["layer"](state["x"], state["ids"], state["weights"])


def work(case):
    op = case["op"]
    if op == "moe":
        t, h, i, e, topk = (case[key] for key in ("tokens", "hidden", "inter", "experts", "topk"))
        experts = e * (1.0 - (1.0 - topk / e) ** t)               # experts that some token is sent to (equal popularity)
        return {"bytes": experts * 3 * h * i * (0.5 + 1 / 16) + t * (4 * h + 12 * topk), "flops": 6.0 * t * topk * h * i}
    if op == "quantize":
        size = {"bf16": 2, "f16": 2, "f32": 4}[case["x"]]
        n = case["rows"] * case["k"]
        return {"bytes": n * (size + 0.5 + (1 / 32 if case["format"] == "mx" else 1 / 16)), "flops": 0}
    m, n, k = case["m"], case["n"], case["k"]
    packed = 0.5 + (1 / 32 if op == "mx_linear" or case.get("format") == "mx" else 1 / 16)
    a = packed if op == "gemm" else {"bf16": 2, "f16": 2, "f32": 4}[case["x"]]
    return {"bytes": m * k * a + n * k * packed + 2 * m * n, "flops": 2.0 * m * n * k}


def tolerance(case):
    op = case["op"]
    if op == "quantize":
        return "exact"
    if op == "moe":
        # Another order of the sums gave the same bits. What may differ is the rounding of an activation to bf16 (the
        # exponential of the SwiGLU is not the same in every implementation) and through it one E2M1 code of the
        # re-quantised activation: with one token that moves a whole row of six experts' sums by up to a step of
        # two block scales in 2048 x 6 terms, 0.9 % of its norm.
        return {"rel": 1e-2, "max": 6e-2}
    # Products of E2M1 codes and E4M3 (or power-of-two) scales have so few significant bits that their FP32 sums came out
    # the same in every order, and equal to the 64-bit product rounded once; what is allowed for is the last place of
    # the output type in a few values.
    return {"rel": 1e-4, "max": 1e-3} if case["out"] == "f16" else {"rel": 8e-4, "max": 8e-3}


# ---- the same results in 64 bits, in plain torch ----------------------------------------------------------------


def _e2m1(q):
    """Quotients -> the nearest E2M1 values (ties to the even code), signs kept, in 64 bits."""
    mag = q.abs().double()
    level = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device=q.device)
    mid = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], dtype=torch.float64, device=q.device)
    code = torch.bucketize(mag, mid)                              # midpoints below the magnitude
    on = mag == mid[code.clamp(max=6)]
    code += on & (code % 2 == 1)
    return torch.where(q < 0, -level[code], level[code])


def _rounded(x, mx):
    """x [rows, K] -> the values its NVFP4 (or MXFP4) form stands for, in 64 bits; by row blocks, to bound the memory."""
    out = torch.empty(x.shape, dtype=torch.float64, device=x.device)
    step = max(1, (1 << 25) // x.shape[1])
    for r in range(0, x.shape[0], step):
        part = x[r:r + step].float()
        blocks = part.reshape(part.shape[0], -1, 32 if mx else 16)
        amax = blocks.abs().amax(-1, keepdim=True)
        if mx:
            scale = torch.exp2((torch.frexp(amax).exponent - 3).double())
        else:
            scale = (amax / 6.0).clamp(2.0 ** -9, 448.0).to(torch.float8_e4m3fn).double()
        out[r:r + step] = (_e2m1(blocks / scale.float()) * scale).reshape(part.shape)
    return out


def _exact_moe(case, gen):
    w1, w2, x, ids, weights = _moe_inputs(case, gen)
    inter = case["inter"]
    x = _rounded(x, False)
    slots = torch.zeros((*ids.shape, case["hidden"]), dtype=torch.float64, device="cuda")
    for e in ids.unique().tolist():
        token, slot = torch.nonzero(ids == e, as_tuple=True)
        gate_up = (x[token] @ _rounded(w1[e], False).T).bfloat16().double()            # the layer's own rounding points
        gate, up = gate_up[:, :inter].clamp(max=10.0), gate_up[:, inter:].clamp(-10.0, 10.0)
        act = (gate * torch.sigmoid(gate) * up * weights[token, slot].double()[:, None]).bfloat16()
        slots[token, slot] = (_rounded(act, False) @ _rounded(w2[e], False).T).bfloat16().double()
    return slots.sum(1)


def exact(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["op"] == "quantize":
        return None                                               # bytes: compared as they are
    if case["op"] == "moe":
        return _exact_moe(case, gen)
    b, x = _product_inputs(case, gen)
    mx = _is_mx(case)
    return _rounded(x, mx) @ _rounded(b, mx).T
