"""The work a program has this framework do, as cases that can be timed: decode steps, quantised projections,
dense products with their fused epilogue, row reductions and sampling, each through the public call a program makes.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call (device tensors, weights, a decoder)
    run(state)          one pass; its outputs
    work(case)          bytes and operations one pass cannot do without
    tolerance(case)     how far two correct evaluations of the same precision may be apart
"""
import importlib
import math

import torch

pkg = importlib.import_module("metal-pjrt-plugin_b200")

DEVICE = "cuda:0"
TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}

# Decoder: the benchmark's layer (hidden 4096, 32 query and 8 KV heads of 128, intermediate 3 x hidden), 6 of its 36
# layers, and a vocabulary cut by about the same factor, so that the LM head keeps its share of the step.
LAYERS, VOCAB, HEAD_DIM = 6, 25600, 128


def listed():
    return [
        # one user talking to the model: the latency of a token, 2048 tokens into the conversation
        dict(name="decode_b1", kind="decode", batch=1, hidden=4096, ctx=2048),
        # a few users served together, in the middle of shorter conversations
        dict(name="decode_b8", kind="decode", batch=8, hidden=4096, ctx=777),
        # the largest decode batch, on full caches
        dict(name="decode_b32", kind="decode", batch=32, hidden=4096, ctx=2048),
        # the smallest call: one token through the fused RMSNorm + qkv projection, int4
        dict(name="linear_int4_m1_qkv", kind="linear", weight="int4", m=1, n=6144, k=4096, form="rms"),
        # the int8 per-channel down projection at the largest decode batch, added to the residual stream
        dict(name="linear_int8_m32_down", kind="linear", weight="int8", m=32, n=4096, k=12288, form="residual"),
        # a prompt of 512 tokens through the largest projection
        dict(name="linear_int4_m512_gate_up", kind="linear", weight="int4", m=512, n=24576, k=4096, form="plain"),
        # a bf16 layer applied to a handful of rows, and to a training-sized batch
        dict(name="gemm_bf16_m16", kind="gemm", dtype="bf16", m=16, n=4096, k=4096, batch=1, layout="nn", act=3, bias=True, aux=False),
        dict(name="gemm_bf16_m8192", kind="gemm", dtype="bf16", m=8192, n=4096, k=4096, batch=1, layout="nn", act=3, bias=True, aux=False),
        # the f32 block of a small model
        dict(name="gemm_f32_m512", kind="gemm", dtype="f32", m=512, n=1024, k=1024, batch=1, layout="nn", act=0, bias=True, aux=False),
        # attention scores q k^T of 32 heads over a ragged sequence
        dict(name="gemm_f16_scores_777", kind="gemm", dtype="f16", m=777, n=777, k=128, batch=32, layout="nt", act=0, bias=False, aux=False),
        # softmax over score rows
        dict(name="softmax_f32_8192x1024", kind="rows", op="softmax", dtype="f32", rows=8192, n=1024),
        # the next token of every sequence of a batch, as chat programs draw it
        dict(name="sample_b32", kind="sample", batch=32, vocab=151936, temperature=0.7, top_k=20, top_p=0.95),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _size(rng, lo, hi):
    """Log-uniform; half of the time as it falls (odd ones among them), half of the time a multiple of 64."""
    v = _log_int(rng, lo, hi)
    return v if rng.random() < 0.5 else max(64, (v + 32) // 64 * 64)


def draw(rng):
    kind = rng.choice(["decode", "decode", "linear", "linear", "gemm", "gemm", "rows", "sample"])
    if kind == "decode":
        return dict(kind=kind, batch=_log_int(rng, 1, 32), hidden=rng.choice([1024, 2048, 4096]), ctx=_log_int(rng, 16, 2048))
    if kind == "linear":
        hidden = rng.choice([1024, 2048, 4096])
        n, k = rng.choice([(hidden, hidden), (hidden // 4, hidden), (hidden + hidden // 2, hidden), (6 * hidden, hidden), (hidden, 3 * hidden)])
        m = _log_int(rng, 1, 1024)
        form = rng.choice(["plain", "residual", "rms"] if m <= 8 else ["plain", "residual"])
        return dict(kind=kind, weight=rng.choice(["int4", "int4", "int8", "int8_g64", "bf16"]), m=m, n=n, k=k, form=form)
    if kind == "gemm":
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        most = 2 ** 32 if dtype == "f32" else 2 ** 37
        while True:
            if rng.random() < 0.25:
                batch, m, n, k = _log_int(rng, 2, 32), _size(rng, 16, 1024), _size(rng, 16, 1024), rng.choice([64, 128, 256])
            else:
                batch, m, n, k = 1, _log_int(rng, 1, 8192), _size(rng, 64, 8192), _size(rng, 64, 8192)
            if batch * m * n * k <= most:
                break
        act, bias = (0, False) if batch > 1 else (rng.choice([0, 1, 2, 3]), rng.random() < 0.5)
        # nn: the layer itself; nt: its gradient towards the input, or scores; tn: its gradient towards the weights
        return dict(kind=kind, dtype=dtype, m=m, n=n, k=k, batch=batch, layout=rng.choice(["nn", "nt", "tn"]), act=act, bias=bias,
                    aux=act != 0 and rng.random() < 0.25)
    if kind == "rows":
        op = rng.choice(["rms", "softmax", "log_softmax", "layernorm"])
        while True:
            rows, n = _log_int(rng, 1, 16384), _size(rng, 64, 16384)
            if rows * n <= 2 ** 25:
                break
        return dict(kind=kind, op=op, dtype=rng.choice(["f32", "bf16"]), rows=rows, n=n)
    way = rng.choice(["greedy", "top_k", "top_p", "all"])
    return dict(kind=kind, batch=_log_int(rng, 1, 32), vocab=rng.choice([32000, 50257, 128256, 151936]),
                temperature=0.0 if way == "greedy" else 0.7, top_k={"top_k": 50, "top_p": 20}.get(way, 0),
                top_p=0.95 if way == "top_p" else 1.0)


# ---- inputs ------------------------------------------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _randn(g, shape, sigma=1.0, dtype=torch.bfloat16):
    return torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32).mul_(sigma).to(dtype)


def _weight(g, n, k, kind):
    w = torch.randn((n, k), generator=g, device=DEVICE, dtype=torch.float32).mul_(0.02)
    if kind == "int4":
        return pkg.qwen3.quantize_int4(w)
    if kind == "int8":
        return pkg.qwen3.quantize_int8(w)
    if kind == "int8_g64":
        return pkg.qwen3.quantize_int8(w, 64)
    return w.to(torch.bfloat16)


def _gain(g, n, dtype=torch.bfloat16):
    return _randn(g, (n,), 0.1, torch.float32).add_(1.0).to(dtype)


def _decoder_config(case):
    heads = case["hidden"] // HEAD_DIM
    return dict(layers=LAYERS, hidden=case["hidden"], heads=heads, kv_heads=heads // 4, head_dim=HEAD_DIM, inter=3 * case["hidden"],
                vocab=VOCAB, theta=1e6, eps=1e-6)


def _prepare_decode(case, g):
    cfg = _decoder_config(case)
    b, ctx, e, d, kv, i = case["batch"], case["ctx"], cfg["hidden"], HEAD_DIM, cfg["kv_heads"], cfg["inter"]
    slots = (ctx + 128) // 128 * 128      # the window rounded up
    layers = []
    for _ in range(LAYERS):
        layers.append({"attn_norm": _gain(g, e), "qkv": _weight(g, (cfg["heads"] + 2 * kv) * d, e, "int4"), "q_norm": _gain(g, d),
                       "k_norm": _gain(g, d), "o": _weight(g, e, e, "int4"), "mlp_norm": _gain(g, e),
                       "gate_up": _weight(g, 2 * i, e, "int4"), "down": _weight(g, e, i, "int4")})
    params = {"embed": _randn(g, (VOCAB, e), 0.02), "layers": layers, "norm": _gain(g, e), "lm_head": _randn(g, (VOCAB, e), 0.02)}
    k = torch.zeros((LAYERS, b, kv, slots, d), dtype=torch.bfloat16, device=DEVICE)
    v = torch.zeros((LAYERS, b, kv, d, slots), dtype=torch.bfloat16, device=DEVICE)
    for layer in range(LAYERS):
        k[layer, :, :, :ctx] = _randn(g, (b, kv, ctx, d))
        v[layer, :, :, :, :ctx] = _randn(g, (b, kv, d, ctx))
    cache = {"k": list(k.unbind(0)), "v": list(v.unbind(0))}
    return {"decoder": pkg.qwen3.Decoder(params, cache, cfg, max_batch=b), "k": k, "v": v,
            "tokens": torch.randint(0, VOCAB, (b,), generator=g, device=DEVICE, dtype=torch.int32),
            "pos": torch.full((1,), ctx, dtype=torch.int32, device=DEVICE),
            "logits": torch.empty((b, VOCAB), dtype=torch.float32, device=DEVICE)}


def _prepare_linear(case, g):
    m, n, k = case["m"], case["n"], case["k"]
    more = {"residual": {"residual": _randn(g, (m, n))}, "rms": {"rms_gain": _gain(g, k)}}.get(case["form"], {})
    return {"x": _randn(g, (m, k)), "w": _weight(g, n, k, case["weight"]), "more": more}


def _prepare_gemm(case, g):
    m, n, k, batch, dtype = case["m"], case["n"], case["k"], case["batch"], TORCH[case["dtype"]]
    ta, tb = case["layout"] == "tn", case["layout"] == "nt"
    # scores of normalised heads, or activations against weights whose product keeps unit variance
    a = _randn(g, (batch, k, m) if ta else (batch, m, k), 1.0, dtype)
    b = _randn(g, (batch, n, k) if tb else (batch, k, n), 1.0 if batch > 1 else k ** -0.5, dtype)
    bias = _randn(g, (n,), 0.01, dtype) if case["bias"] else None
    state = {"a": a, "b": b, "bias": bias, "act": case["act"], "tb": tb}
    if batch == 1 and not ta and not case["aux"]:
        return dict(state, a=a[0], b=b[0])           # a plain layer: blas.matmul
    d = torch.empty((batch, m, n), dtype=dtype, device=DEVICE)
    aux = torch.empty_like(d) if case["aux"] else None
    B = pkg.blas
    p = B.GemmParams(m, n, k, B.Operand(a, a.stride(1), a.stride(0), ta), B.Operand(b, b.stride(1), b.stride(0), tb),
                     B.Operand(d, d.stride(1), d.stride(0)), batch, alpha=k ** -0.5 if batch > 1 else 1.0)
    return dict(state, params=p, epilogue=B.SteelEpilogue(case["act"], bias, aux), d=d, aux=aux)


def _prepare_rows(case, g):
    dtype = TORCH[case["dtype"]]
    sigma = 3.0 if "softmax" in case["op"] else 1.0
    return {"op": case["op"], "x": _randn(g, (case["rows"], case["n"]), sigma, dtype), "gain": _gain(g, case["n"], dtype),
            "beta": _randn(g, (case["n"],), 0.1, dtype)}


def _prepare_sample(case, g):
    kw = dict(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"])
    return {"logits": _randn(g, (case["batch"], case["vocab"]), 3.0, torch.float32), "kw": kw,
            "uniform": torch.rand((case["batch"],), generator=g, device=DEVICE)}


_PREPARE = {"decode": _prepare_decode, "linear": _prepare_linear, "gemm": _prepare_gemm, "rows": _prepare_rows, "sample": _prepare_sample}


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, _generator(seed)), kind=case["kind"])


# ---- one pass ----------------------------------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "decode":
        logits = state["decoder"].step(state["tokens"], state["pos"], state["logits"])
        return {"logits": logits, "k": state["k"], "v": state["v"]}
    if kind == "linear":
        return pkg.qwen3.linear(state["x"], state["w"], **state["more"])
    if kind == "gemm":
        if "params" in state:
            pkg.blas.run_steel_gemm(state["params"], state["epilogue"])
            return {"d": state["d"], "aux": state["aux"]}
        return pkg.blas.matmul(state["a"], state["b"], state["bias"], state["act"], transpose_b=state["tb"])
    if kind == "rows":
        op, x = state["op"], state["x"]
        if op == "rms":
            return pkg.rows.rms_norm(x, state["gain"], 1e-6)
        if op == "layernorm":
            return pkg.rows.layer_norm(x, state["gain"], state["beta"])
        return pkg.rows.softmax(x) if op == "softmax" else pkg.rows.log_softmax(x)
    return pkg.qwen3.sample(state["logits"], state["uniform"], **state["kw"])


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------

BYTES_PER_WEIGHT = {"int4": 0.5 + 4 / 64, "int8": 1.0, "int8_g64": 1.0 + 2 / 64, "bf16": 2.0}
ELEMENT = {"f32": 4, "f16": 2, "bf16": 2}


def work(case):
    kind = case["kind"]
    if kind == "decode":
        cfg = _decoder_config(case)
        b, e, d, kv, i = case["batch"], cfg["hidden"], HEAD_DIM, cfg["kv_heads"], cfg["inter"]
        weights = LAYERS * ((cfg["heads"] + 2 * kv) * d * e + e * e + 3 * i * e)
        slots = LAYERS * b * 2 * kv * d * (case["ctx"] + 1)          # K and V rows read, the new ones among them
        return {"bytes": weights * BYTES_PER_WEIGHT["int4"] + VOCAB * e * 2 + slots * 2 + b * (e * 2 + VOCAB * 4),
                "flops": 2 * b * (weights + VOCAB * e) + 2 * slots * (cfg["heads"] // kv)}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        extra = {"residual": 2 * m * n, "rms": 2 * k}.get(case["form"], 0) + (2 * n if case["weight"] == "int8" else 0)
        return {"bytes": n * k * BYTES_PER_WEIGHT[case["weight"]] + 2 * m * (n + k) + extra, "flops": 2 * m * n * k}
    if kind == "gemm":
        m, n, k, batch = case["m"], case["n"], case["k"], case["batch"]
        values = batch * (m * k + k * n + m * n * (2 if case["aux"] else 1)) + (n if case["bias"] else 0)
        return {"bytes": values * ELEMENT[case["dtype"]], "flops": 2 * batch * m * n * k}
    if kind == "rows":
        values = case["rows"] * case["n"]
        vectors = case["n"] * {"rms": 1, "layernorm": 2}.get(case["op"], 0)
        return {"bytes": (2 * values + vectors) * ELEMENT[case["dtype"]], "flops": 5 * values}
    return {"bytes": case["batch"] * (case["vocab"] * 4 + 8), "flops": 2 * case["batch"] * case["vocab"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "decode":
        # a bf16 activation that rounds the other way moves every value after it a little; six layers of that
        return {"rel": 2.5e-2}
    if kind == "linear":
        return {"rel": 1e-2}              # bf16 results; for many rows the weights are bf16 before the product
    if kind == "gemm":
        return {"rel": {"f32": 1e-5, "f16": 2e-3, "bf16": 1e-2}[case["dtype"]]}
    if kind == "rows":
        return {"rel": {"f32": 1e-5, "bf16": 1e-2}[case["dtype"]]}
    return "exact"
