"""The work a user of this package has it do, as timed cases.

Five kinds of pass, all through the package's public entry points:

* ``call``  one decode-matmul as a model's host code issues it: quantised weight resident and
            repacked, activations in hand, the result a new tensor.  Every weight format, any batch.
* ``step``  the linears of several transformer layers at a decode batch size, captured once in a
            CUDA graph with launch overlap on and replayed for every token, as a serving loop does.
* ``mlp``   a gated MLP with int8 per-channel weights: gate/up with the fused activation, then down.
* ``moe``   an expert layer: route, gather, two grouped matmuls, weighted combine.
* ``load``  bringing a weight into the kernels' layout when a model is loaded: quantise + repack of
            an fp16 weight, or the repack of one that is already packed.

Weights are resident and repacked before a pass (``prepare``), as parameters are in use.  Values
follow the benchmark's distributions: activations N(0, 1), uniform codes, scales U(0.001, 0.01)
for int4 and U(1e-4, 1e-3) for int8.
"""
import math

import torch

import relax_b200
from relax_b200 import ops, patterns

DEV = "cuda"

PATTERN_OF_EPILOGUE = {
    "none": "cutlass.decode_matmul",
    "bias": "cutlass.decode_matmul_bias",
    "bias_gelu": "cutlass.decode_matmul_bias_gelu",
    "bias_add": "cutlass.decode_matmul_bias_residual_add",
    "bias_mul_relu": "cutlass.decode_matmul_bias_residual_multiply_relu",
}


def listed():
    return [
        # one projection for one sequence: what an interactive session issues between two tokens,
        # where latency and launch count are everything
        dict(name="call_q4_m1", kind="call", fmt="q4", m=1, k=4096, n=4096, group=32, epilogue="none"),
        # an act-order AutoGPTQ checkpoint (fp16 zero points, activations gathered first), four sequences
        dict(name="call_gptq_m4", kind="call", fmt="gptq", m=4, k=4096, n=11008, group=128, epilogue="bias"),
        # an output projection whose width is no multiple of a tile, for a serving batch just above
        # the small-batch range
        dict(name="call_ft8_m48_ragged", kind="call", fmt="ft8", m=48, k=4096, n=32016, group=-1, epilogue="bias"),
        # the linears of four Llama-2-7B layers (weights far larger than L2), one sequence and a full
        # decode batch
        dict(name="step_q4_m1", kind="step", m=1, layers=4, hidden=4096, ffn=11008, group=32, zeros=False),
        dict(name="step_q4_m32", kind="step", m=32, layers=4, hidden=4096, ffn=11008, group=32, zeros=False),
        # a 2048-token prompt through the widest linear, group-128 scales and zero points
        dict(name="call_q4z_m2048", kind="call", fmt="q4z", m=2048, k=4096, n=22016, group=128, epilogue="none"),
        # the Llama-70B MLP in int8: a decode batch, a short prompt, and a long one (the largest case)
        dict(name="mlp_ft8_m16", kind="mlp", m=16, hidden=8192, ffn=28672),
        dict(name="mlp_ft8_m256", kind="mlp", m=256, hidden=8192, ffn=28672),
        dict(name="mlp_ft8_m4096", kind="mlp", m=4096, hidden=8192, ffn=28672),
        # the Mixtral-shaped expert layer: eight sequences decoding, and a 512-token prompt
        dict(name="moe_ft4_t8", kind="moe", fmt="ft4", tokens=8, hidden=4096, ffn=14336, experts=8, top_k=2, group=128),
        dict(name="moe_ft4_t512", kind="moe", fmt="ft4", tokens=512, hidden=4096, ffn=14336, experts=8, top_k=2, group=128),
        # quantising and repacking one fp16 weight at load time
        dict(name="load_fp16_ft4", kind="load", src="fp16", bits=4, group=-1, k=4096, n=11008),
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, int(v / step) * step)


def draw(rng):
    kind = rng.choice(["call", "call", "step", "mlp", "moe", "load"])
    if kind == "call":
        fmt = rng.choice(["q4", "gptq", "ft4", "q4z", "ft8", "ft8g"])
        m = _log_int(rng, 1, 2048)
        k = _log_int(rng, 1024, 14336, 128)
        n = _log_int(rng, 1024, 32768, rng.choice([16, 128]))
        group = {"q4": rng.choice([32, 64, 128]), "gptq": 128, "ft4": -1, "q4z": rng.choice([32, 64, 128]), "ft8": -1, "ft8g": 64}[fmt]
        epilogue = rng.choice(["none", "bias", "bias_gelu", "bias_add", "bias_mul_relu"])
        if fmt == "gptq":
            epilogue = rng.choice(["none", "bias"])
        return dict(kind=kind, fmt=fmt, m=m, k=k, n=n, group=group, epilogue=epilogue)
    if kind == "step":
        hidden = rng.randrange(2048, 5121, 256)
        ffn = int(hidden * rng.uniform(2.0, 3.5)) // 128 * 128
        return dict(kind=kind, m=_log_int(rng, 1, 32), layers=rng.randint(2, 4), hidden=hidden, ffn=ffn,
                    group=rng.choice([32, 32, 128]), zeros=rng.choice([False, False, True]))
    if kind == "mlp":
        hidden = rng.randrange(2048, 8193, 256)
        ffn = int(hidden * rng.uniform(1.0, 3.5)) // 128 * 128
        return dict(kind=kind, m=_log_int(rng, 1, 4096), hidden=hidden, ffn=ffn)
    if kind == "moe":
        fmt = rng.choice(["ft4", "ft8", "fp16"])
        hidden = rng.randrange(1024, 4097, 256)
        ffn = int(hidden * rng.uniform(1.0, 3.5)) // 128 * 128
        return dict(kind=kind, fmt=fmt, tokens=_log_int(rng, 1, 1024), hidden=hidden, ffn=ffn,
                    experts=rng.choice([4, 8, 16]), top_k=rng.choice([1, 2, 4]), group=-1 if fmt != "ft4" else 128)
    src = rng.choice(["fp16", "q4", "gptq", "ft"])
    bits = rng.choice([4, 8]) if src in ("fp16", "ft") else 4
    group = rng.choice([-1, 64]) if src == "fp16" and bits == 8 else -1
    return dict(kind=kind, src=src, bits=bits, group=group, k=_log_int(rng, 1024, 14336, 128),
                n=_log_int(rng, 1024, 28672, rng.choice([32, 128])))


# ------------------------------------------------------------------ inputs

def _rand_half(g, shape, lo, hi):
    return (torch.rand(shape, device=DEV, generator=g) * (hi - lo) + lo).half()


def _normal(g, *shape):
    return torch.randn(shape, device=DEV, generator=g, dtype=torch.float32).half()


def _bytes(g, *shape):
    return torch.randint(-128, 128, shape, dtype=torch.int8, device=DEV, generator=g)


def _words(g, *shape):
    return torch.randint(-2 ** 31, 2 ** 31 - 1, shape, dtype=torch.int32, device=DEV, generator=g)


def _groups(c):
    return 1 if c["group"] <= 0 else c["k"] // c["group"]


def prepare(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return {"call": _prepare_call, "step": _prepare_step, "mlp": _prepare_mlp, "moe": _prepare_moe,
            "load": _prepare_load}[case["kind"]](case, g)


def _prepare_call(c, g):
    m, k, n, fmt = c["m"], c["k"], c["n"], c["fmt"]
    s = {"case": c, "x": _normal(g, m, k), "bias": None, "residual": None}
    if c["epilogue"] != "none":
        s["bias"] = _normal(g, n)
    if c["epilogue"] in ("bias_add", "bias_mul_relu"):
        s["residual"] = _normal(g, m, n)
    if fmt == "q4":
        s["w"] = ops.preprocess_weight_q4f16(_words(g, n, k // 8))
        s["scales"] = _rand_half(g, (n, k // c["group"]), 0.001, 0.01)
    elif fmt == "gptq":
        groups = _groups(c)
        order = torch.randperm(k, device=DEV, generator=g)
        g_idx = (torch.arange(k, device=DEV) // c["group"])[order].to(torch.int32)
        s["perm"] = ops.gptq_act_order(g_idx, groups)
        s["w"] = ops.preprocess_weight_autogptq(_words(g, k // 8, n), s["perm"])
        s["zeros"] = ops.unpack_zeros_autogptq(_words(g, groups, n // 8))
        s["scales"] = _rand_half(g, (groups, n), 0.001, 0.01)
    elif fmt == "q4z":
        s["w"] = ops.preprocess_weight_q4f16(_words(g, n, k // 8))
        s["scales"] = _rand_half(g, (n, k // c["group"]), 0.001, 0.01)
        s["zeros"] = torch.randint(0, 16, (n, k // c["group"]), device=DEV, generator=g).half()
    else:
        bits = 4 if fmt == "ft4" else 8
        s["w"] = ops.preprocess_weight_ft(_bytes(g, k, n // 2 if bits == 4 else n), bits == 4)
        lo, hi = (0.001, 0.01) if bits == 4 else (1e-4, 1e-3)
        s["scales"] = _rand_half(g, (n,) if c["group"] <= 0 else (k // c["group"], n), lo, hi)
    return s


def _prepare_step(c, g):
    m, h, f, gs = c["m"], c["hidden"], c["ffn"], c["group"]

    def linear(n, k, gated=False):
        w = _words(g, n, k // 8)
        w = ops.preprocess_weight_gate_up(w) if gated else ops.preprocess_weight_q4f16(w)
        sc = _rand_half(g, (n, k // gs), 0.001, 0.01)
        z = torch.randint(0, 16, (n, k // gs), device=DEV, generator=g).half() if c["zeros"] else None
        if gated:
            sc = ops.interleave_gate_up(sc)
            z = ops.interleave_gate_up(z) if z is not None else None
        return w, sc, z

    layers = []
    for _ in range(c["layers"]):
        layers.append(dict(
            qkv=linear(3 * h, h), o=linear(h, h), gate_up=linear(2 * f, h, True), down=linear(h, f),
            x=_normal(g, m, h), attn=_normal(g, m, h), xm=_normal(g, m, h),
            out_qkv=torch.empty(m, 3 * h, dtype=torch.float16, device=DEV),
            out_o=torch.empty(m, h, dtype=torch.float16, device=DEV),
            act=torch.empty(m, f, dtype=torch.float16, device=DEV),
            out=torch.empty(m, h, dtype=torch.float16, device=DEV)))

    def one(x, lin, out, activation="identity"):
        ops.gemm_fp16_q4f16(x, lin[0], lin[1], lin[2], activation=activation, group_size=gs, out=out)

    def step():
        for l in layers:
            one(l["x"], l["qkv"], l["out_qkv"])
            one(l["attn"], l["o"], l["out_o"])
            one(l["xm"], l["gate_up"], l["act"], "swiglu")
            one(l["act"], l["down"], l["out"])

    step()  # scratch and module state exist before the capture
    torch.cuda.synchronize()
    before = relax_b200.get_launch_overlap()
    relax_b200.set_launch_overlap(True)
    try:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
    finally:
        relax_b200.set_launch_overlap(before)
    return {"case": c, "graph": graph, "layers": layers,
            "outs": [(l["out_qkv"], l["out_o"], l["act"], l["out"]) for l in layers]}


def _prepare_mlp(c, g):
    h, f = c["hidden"], c["ffn"]
    gate_up = torch.randint(-127, 128, (h, 2 * f), dtype=torch.int8, device=DEV, generator=g)
    down = torch.randint(-127, 128, (f, h), dtype=torch.int8, device=DEV, generator=g)
    return {"case": c, "x": _normal(g, c["m"], h),
            "gate_up": ops.preprocess_weight_gate_up(gate_up, ops.LAYOUT_FT_KN, False),
            "gate_up_s": ops.interleave_gate_up(_rand_half(g, (2 * f,), 1e-4, 1e-3)),
            "down": ops.preprocess_weight_ft(down, False), "down_s": _rand_half(g, (h,), 1e-4, 1e-3)}


def _prepare_moe(c, g):
    h, f, e = c["hidden"], c["ffn"], c["experts"]
    s = {"case": c, "x": _normal(g, c["tokens"], h), "logits": torch.randn(c["tokens"], e, device=DEV, generator=g)}
    for name, k, n, hi in (("1", h, f, 0.01), ("2", f, h, 0.001)):
        if c["fmt"] == "fp16":
            w = torch.empty(e, n, k, dtype=torch.float16, device=DEV)
            for i in range(e):
                w[i] = _normal(g, n, k) * (2.0 / math.sqrt(k))
            s["w" + name] = w
            continue
        bits = 4 if c["fmt"] == "ft4" else 8
        s["w" + name] = ops.preprocess_weight_ft(_bytes(g, e, k, n // 2 if bits == 4 else n), bits == 4)
        hi = hi if bits == 4 else hi / 10
        s["s" + name] = _rand_half(g, (e, n) if c["group"] <= 0 else (e, k // c["group"], n), hi / 10, hi)
    return s


def _prepare_load(c, g):
    k, n = c["k"], c["n"]
    s = {"case": c}
    if c["src"] == "fp16":
        s["w"] = _normal(g, n, k) * 0.02
    elif c["src"] == "q4":
        s["w"] = _words(g, n, k // 8)
    elif c["src"] == "gptq":
        s["w"] = _words(g, k // 8, n)
        s["zeros"] = _words(g, k // 128, n // 8)
    else:
        s["w"] = _bytes(g, k, n // 2 if c["bits"] == 4 else n)
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    return {"call": _run_call, "step": _run_step, "mlp": _run_mlp, "moe": _run_moe, "load": _run_load}[s["case"]["kind"]](s)


def _run_call(s):
    c = s["case"]
    fmt = c["fmt"]
    if fmt == "gptq":
        return ops.gemm_fp16_autogptq(s["x"], s["w"], s["scales"], s["zeros"], bias=s["bias"], perm=s["perm"])
    if fmt in ("q4", "q4z"):
        e = c["epilogue"]
        return ops.gemm_fp16_q4f16(s["x"], s["w"], s["scales"], zeros=s.get("zeros"), bias=s["bias"], residual=s["residual"],
                                   activation="gelu" if e == "bias_gelu" else "identity",
                                   binary_op={"bias_add": "plus", "bias_mul_relu": "multiply"}.get(e, ""),
                                   unary_op="relu" if e == "bias_mul_relu" else "identity", group_size=c["group"])
    return patterns.run_pattern(PATTERN_OF_EPILOGUE[c["epilogue"]], s["x"], s["w"], s["scales"], s["bias"], s["residual"])


def _run_step(s):
    s["graph"].replay()
    return s["outs"]


def _run_mlp(s):
    h = ops.gemm_fp16_ft(s["x"], s["gate_up"], s["gate_up_s"], 8, activation="swiglu")
    return h, ops.gemm_fp16_ft(h, s["down"], s["down_s"], 8)


def _run_moe(s):
    c = s["case"]
    indptr, token_of_row, gate_of_row, row_of_flat = ops.moe_route(s["logits"], c["top_k"])
    xg = ops.moe_gather(s["x"], token_of_row)
    if c["fmt"] == "fp16":
        y = ops.group_gemm_fp16(xg, s["w1"], indptr)
        y = ops.group_gemm_fp16(y, s["w2"], indptr)
    else:
        y = ops.moe_gemm_ft(xg, s["w1"], s["s1"], indptr)
        y = ops.moe_gemm_ft(y, s["w2"], s["s2"], indptr)
    return ops.moe_combine(y, row_of_flat, gate_of_row, c["top_k"]), indptr, token_of_row, gate_of_row, row_of_flat


def _run_load(s):
    c = s["case"]
    if c["src"] == "fp16":
        packed, scales = ops.encode_ft(s["w"], c["bits"], c["group"])
        return ops.preprocess_weight_ft(packed, c["bits"] == 4), scales
    if c["src"] == "q4":
        return ops.preprocess_weight_q4f16(s["w"])
    if c["src"] == "gptq":
        return ops.preprocess_weight_autogptq(s["w"]), ops.unpack_zeros_autogptq(s["zeros"])
    return ops.preprocess_weight_ft(s["w"], c["bits"] == 4)


# ------------------------------------------------------------------ what a pass cannot do without

def _linear_bytes(m, k, n, bits, groups, zeros=False):
    return n * k * bits / 8 + n * groups * 2 * (2 if zeros else 1) + m * k * 2 + m * n * 2


def work(case):
    c = case
    if c["kind"] == "call":
        bits = 8 if c["fmt"] in ("ft8", "ft8g") else 4
        m, k, n = c["m"], c["k"], c["n"]
        b = _linear_bytes(m, k, n, bits, _groups(c), c["fmt"] in ("gptq", "q4z"))
        b += n * 2 * (c["epilogue"] != "none") + m * n * 2 * (c["epilogue"] in ("bias_add", "bias_mul_relu"))
        b += k * 4 * (c["fmt"] == "gptq")
        return {"bytes": b, "flops": 2.0 * m * n * k}
    if c["kind"] == "step":
        m, h, f, gs = c["m"], c["hidden"], c["ffn"], c["group"]
        shapes = [(h, 3 * h, 3 * h), (h, h, h), (h, 2 * f, f), (f, h, h)]
        b = sum(_linear_bytes(m, k, n, 4, k // gs, c["zeros"]) - m * (n - n_out) * 2 for k, n, n_out in shapes)
        return {"bytes": c["layers"] * b, "flops": c["layers"] * sum(2.0 * m * k * n for k, n, _ in shapes)}
    if c["kind"] == "mlp":
        m, h, f = c["m"], c["hidden"], c["ffn"]
        return {"bytes": 3.0 * h * f + (2 * f + h) * 2 + 2.0 * m * (2 * h + 2 * f), "flops": 6.0 * m * h * f}
    if c["kind"] == "moe":
        h, f, e, rows = c["hidden"], c["ffn"], c["experts"], c["tokens"] * c["top_k"]
        # experts that some token is routed to (an even spread): only their weights are needed
        used = e * (1.0 - (1.0 - 1.0 / e) ** rows)
        bits = {"ft4": 4, "ft8": 8, "fp16": 16}[c["fmt"]]
        scales = 0 if bits == 16 else 2 * ((h // c["group"]) * f + (f // c["group"]) * h if c["group"] > 0 else f + h)
        b = used * (2.0 * h * f * bits / 8 + scales) + c["tokens"] * (e * 4 + h * 4) + 2.0 * rows * 2 * f
        return {"bytes": b, "flops": 4.0 * rows * h * f}
    k, n = c["k"], c["n"]
    packed = n * k * c["bits"] / 8
    if c["src"] == "fp16":
        groups = 1 if c["group"] <= 0 else k // c["group"]
        return {"bytes": n * k * 2 + packed + groups * n * 2, "flops": 0}
    extra = (k // 128) * n * 2.5 if c["src"] == "gptq" else 0
    return {"bytes": 2 * packed + extra, "flops": 0}


def tolerance(case):
    if case["kind"] == "load":
        return "exact"
    # fp16 results of fp32 sums: half an ulp (2^-12 of the value on average) flips where the order
    # of the sum differs; chained matmuls carry one rounded intermediate
    return {"rel": 1e-3 if case["kind"] == "call" else 2e-3, "differ": 0.0}
