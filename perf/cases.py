"""The work that users of this library have it do, as cases to measure: decode steps, prefill chunks, dense FFNs and routed-MoE
layers, in NVFP4 and FP8, through eider_b200.ops.

Layer sizes are those of the benchmark and of the test suite: hidden 5120 with an FFN of 13824 and a fused QKV of 7168, and
routed layers of 128 experts, top-8, hidden 2048, expert intermediate 768; other sizes are generic ones around them.
Weights are N(0, 0.02^2), activations and router logits N(0, 1): the distributions of the benchmark's configurations.
"""
import math

import torch

from eider_b200 import ops

LISTED = [
    # One user's decode step: every linear is a GEMV that streams its weights once, four FFN layers (gate/up-sized, then
    # down) chained as a model chains them and replayed as one CUDA graph, as the reference replays its decode step.
    {"name": "decode_1", "kind": "decode", "tokens": 1, "hidden": 5120, "inter": 13824, "layers": 4, "dtype": "bf16"},
    # The same step for a batch of 32 running sequences.
    {"name": "decode_32", "kind": "decode", "tokens": 32, "hidden": 5120, "inter": 13824, "layers": 4, "dtype": "bf16"},
    # FP8 attention projections (fused QKV) of eight layers in a batched decode step of eight sequences.
    {"name": "decode_fp8_8", "kind": "decode_fp8", "tokens": 8, "k": 5120, "n": 7168, "layers": 8},
    # One token through four routed-MoE layers (router, top-8 experts, shared expert, residual).
    {"name": "decode_moe", "kind": "decode_moe", "hidden": 2048, "inter": 768, "experts": 128, "top_k": 8, "layers": 4},
    # The smallest call: one linear on one f32 activation row, launched on its own from the host.
    {"name": "one_linear", "kind": "linear", "tokens": 1, "k": 2048, "n": 1536, "dtype": "f32"},
    # The benchmark's prefill chunk: 512 tokens quantized on the fly, then the W4A4 GEMM of a fused gate/up projection.
    {"name": "prefill_512", "kind": "prefill", "tokens": 512, "k": 5120, "n": 27648, "producer": "row", "dtype": "bf16", "out": "bf16"},
    # A ragged last chunk of a prompt through the pre-attention norm and a calibrated QKV projection, f32 results.
    {"name": "norm_qkv_333", "kind": "prefill", "tokens": 333, "k": 5120, "n": 7168, "producer": "norm", "dtype": "f32", "out": "f32"},
    # The largest chunk of the benchmark's sweep through the down projection.
    {"name": "prefill_16384", "kind": "prefill", "tokens": 16384, "k": 13824, "n": 5120, "producer": "row", "dtype": "bf16", "out": "bf16"},
    # FP8 attention projection of a 2048-token chunk, quantized per token on the fly.
    {"name": "prefill_fp8_2048", "kind": "prefill_fp8", "tokens": 2048, "k": 5120, "n": 7168},
    # The whole dense gated FFN of a 512-token chunk with its residual.
    {"name": "ffn_512", "kind": "ffn", "tokens": 512, "hidden": 5120, "inter": 13824, "dtype": "bf16"},
    # The routed-MoE layer of the benchmark: 4096 tokens, 128 experts, top-8.
    {"name": "moe_4096", "kind": "moe", "tokens": 4096, "experts": 128, "top_k": 8, "hidden": 2048, "inter": 768, "dtype": "bf16", "interleaved": True},
    # A short ragged prompt through the same layer: most experts see a handful of rows.
    {"name": "moe_77", "kind": "moe", "tokens": 77, "experts": 128, "top_k": 8, "hidden": 2048, "inter": 768, "dtype": "bf16", "interleaved": True},
]


def listed():
    return [dict(c) for c in LISTED]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def _multiple(rng, lo, hi, step):
    return max(lo, min(hi, _log_int(rng, lo, hi) // step * step))


def draw(rng):
    """One more case: any kind, sizes spread over the range (over its logarithm), token counts of every residue."""
    kind = rng.choice(["decode", "decode_fp8", "decode_moe", "linear", "prefill", "prefill", "prefill_fp8", "ffn", "ffn", "moe", "moe"])
    if kind == "decode":
        tokens = _log_int(rng, 1, 64)
        return {"kind": kind, "tokens": tokens, "hidden": _multiple(rng, 2048, 5120, 128), "inter": _multiple(rng, 4096, 13824, 128),
                "layers": 4, "dtype": rng.choice(["bf16", "bf16", "f32"]) if tokens <= 32 else "bf16"}
    if kind == "decode_fp8":
        return {"kind": kind, "tokens": _log_int(rng, 1, 64), "k": _multiple(rng, 2048, 8192, 128), "n": _multiple(rng, 1024, 8192, 64), "layers": 8}
    if kind == "decode_moe":
        return {"kind": kind, "hidden": _multiple(rng, 1024, 4096, 128), "inter": _multiple(rng, 384, 1536, 64),
                "experts": rng.choice([32, 64, 128]), "top_k": rng.choice([4, 6, 8]), "layers": 4}
    if kind == "linear":
        return {"kind": kind, "tokens": _log_int(rng, 1, 8), "k": _multiple(rng, 1024, 5120, 64), "n": _multiple(rng, 512, 8192, 16),
                "dtype": rng.choice(["bf16", "f32"])}
    if kind == "prefill":
        k, n = rng.choice([(5120, 27648), (5120, 7168), (13824, 5120), (2048, 6144), (4096, 24576), (12288, 4096)])
        most = 16384 if n * k <= 13824 * 5120 else 8192
        producer = rng.choice(["row", "row", "norm", "static"])
        return {"kind": kind, "tokens": _log_int(rng, 17, most), "k": k, "n": n, "producer": producer,
                "dtype": "f32" if producer == "norm" else rng.choice(["bf16", "bf16", "f32"]), "out": rng.choice(["bf16", "bf16", "f32"])}
    if kind == "prefill_fp8":
        return {"kind": kind, "tokens": _log_int(rng, 17, 8192), "k": _multiple(rng, 2048, 8192, 128), "n": _multiple(rng, 1024, 14336, 64)}
    if kind == "ffn":
        hidden, inter = rng.choice([(5120, 13824), (2048, 6144), (4096, 12288)])
        return {"kind": kind, "tokens": _log_int(rng, 17, 4096), "hidden": hidden, "inter": inter, "dtype": rng.choice(["bf16", "bf16", "f32"])}
    return {"kind": kind, "tokens": _log_int(rng, 17, 6144), "experts": rng.choice([64, 128]), "top_k": rng.choice([4, 6, 8]),
            "hidden": rng.choice([1024, 2048, 4096]), "inter": rng.choice([512, 768, 1024]), "dtype": rng.choice(["bf16", "bf16", "f32"]),
            "interleaved": rng.choice([True, True, False])}


# ---- inputs ------------------------------------------------------------------------------------------------
_DTYPE = {"bf16": torch.bfloat16, "f32": torch.float32}


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, shape, dtype=torch.float32, std=1.0):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32).mul_(std).to(dtype)


def _nvfp4_weight(g, n, k, input_scale=1.0):
    # (the checkpoint's global scale: amax / (6 * 448) of N(0, 0.02^2) weights)
    return ops.ModelOptWeight.quantize(_normal(g, (n, k), std=0.02), input_scale=input_scale)


def _experts(g, experts, n, k):
    """Stacked expert weights, quantized one expert at a time."""
    parts = []
    for _ in range(experts):
        parts.append(ops.ModelOptWeight.quantize(_normal(g, (n, k), std=0.02), global_scale=0.1 / 2688.0))
    return parts


def _grouped(g, experts, n, k):
    parts = _experts(g, experts, n, k)
    return ops.GroupedNvfp4Weights.from_checkpoint(
        torch.stack([w.packed for w in parts]), torch.stack([w.scales_row_major for w in parts]),
        torch.full((experts,), parts[0].weight_scale_2, dtype=torch.float32, device="cuda"))


def _captured(step):
    """A decode step as one CUDA graph, as the decode loop keeps it: warmed up once, then captured."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outputs = step()
    return graph, outputs


def prepare(case, seed):
    g = _rng(seed)
    kind = case["kind"]
    if kind == "decode":
        t, h, i, dtype = case["tokens"], case["hidden"], case["inter"], _DTYPE[case["dtype"]]
        x = _normal(g, (t, h), dtype)
        layers = [(_nvfp4_weight(g, i, h), _nvfp4_weight(g, h, i)) for _ in range(case["layers"])]
        up_plan, down_plan = ops.Nvfp4DecodePlan(t, i, h), ops.Nvfp4DecodePlan(t, h, i)
        mid = [torch.empty(t, i, dtype=dtype, device="cuda") for _ in layers]
        out = [torch.empty(t, h, dtype=dtype, device="cuda") for _ in layers]

        def step():
            y = x
            for (up, down), m, o in zip(layers, mid, out):
                y = down_plan.run(up_plan.run(y, up, out=m), down, out=o)
            return mid + out
        graph, outputs = _captured(step)
        return {"kind": "graph", "graph": graph, "outputs": outputs, "keep": (x, layers, up_plan, down_plan)}
    if kind == "decode_fp8":
        t, k, n = case["tokens"], case["k"], case["n"]
        xs = [_normal(g, (t, k), torch.bfloat16) for _ in range(case["layers"])]
        ws = [ops.quantize_fp8_weight(_normal(g, (n, k), std=0.02)) for _ in xs]
        plan = ops.Fp8DecodePlan(t, n, k)
        outs = [torch.empty(t, n, dtype=torch.bfloat16, device="cuda") for _ in xs]

        def step():
            return [plan.run(x, w, s, out=o) for x, (w, s), o in zip(xs, ws, outs)]
        graph, outputs = _captured(step)
        return {"kind": "graph", "graph": graph, "outputs": outputs, "keep": (xs, ws, plan)}
    if kind == "decode_moe":
        h, i, e = case["hidden"], case["inter"], case["experts"]
        layers = [ops.DecodeMoe(_experts(g, e, 2 * i, h), _experts(g, e, h, i), case["top_k"]) for _ in range(case["layers"])]
        xs = [_normal(g, (h,)) for _ in layers]
        logits = [_normal(g, (e,)) for _ in layers]
        shared = [(_normal(g, (1,)), _normal(g, (h,))) for _ in layers]
        residual = _normal(g, (h,))

        def step():
            y, outs = residual, []
            for layer, x, lg, (gate, sh) in zip(layers, xs, logits, shared):
                y = layer.run(x, lg, gate, sh, y)
                outs.append(y)
            return outs
        graph, outputs = _captured(step)
        return {"kind": "graph", "graph": graph, "outputs": outputs, "keep": (layers, xs, logits, shared, residual)}
    if kind == "linear":
        t, k, n = case["tokens"], case["k"], case["n"]
        return {"kind": kind, "x": _normal(g, (t, k), _DTYPE[case["dtype"]]), "w": _nvfp4_weight(g, n, k), "plan": ops.Nvfp4DecodePlan(t, n, k),
                "out": _DTYPE[case["dtype"]]}
    if kind == "prefill":
        t, k, n = case["tokens"], case["k"], case["n"]
        # a calibrated input scale spreads N(0, 1) activations over the block scales: amax / (6 * 448), amax = 4.5
        scale = 1.0 if case["producer"] == "row" else 4.5 / 2688.0
        return {"kind": kind, "producer": case["producer"], "x": _normal(g, (t, k), _DTYPE[case["dtype"]]), "w": _nvfp4_weight(g, n, k, scale),
                "norm": _normal(g, (k,), std=0.1).add_(1.0) if case["producer"] == "norm" else None,
                "plan": ops.Fp4TnMatmulPlan(t, n, k), "out": _DTYPE[case["out"]]}
    if kind == "prefill_fp8":
        t, k, n = case["tokens"], case["k"], case["n"]
        return {"kind": kind, "x": _normal(g, (t, k), torch.bfloat16), "w": ops.quantize_fp8_weight(_normal(g, (n, k), std=0.02)),
                "plan": ops.Fp8TnMatmulPlan(t, n, k)}
    if kind == "ffn":
        t, h, i = case["tokens"], case["hidden"], case["inter"]
        # gate and up are about 0.02 * sqrt(hidden) wide each, their SiLU product reaches some 20 times that
        ffn = ops.DenseFfn(_nvfp4_weight(g, 2 * i, h), _nvfp4_weight(g, h, i, 20.0 / 2688.0))
        ffn.plans(t)
        return {"kind": kind, "ffn": ffn, "x": _normal(g, (t, h), _DTYPE[case["dtype"]]), "residual": _normal(g, (t, h), torch.bfloat16)}
    if kind == "moe":
        t, e, h, i = case["tokens"], case["experts"], case["hidden"], case["inter"]
        gate_up, down = _grouped(g, e, 2 * i, h), _grouped(g, e, h, i)
        return {"kind": kind, "moe": ops.GroupedMoe(t, e, case["top_k"], h, i), "x": _normal(g, (t, h), _DTYPE[case["dtype"]]),
                "logits": _normal(g, (t, e)), "gate_up": gate_up, "down": down,
                "interleaved": gate_up.interleave_gate_up() if case["interleaved"] else None}
    raise ValueError(kind)


def run(state):
    kind = state["kind"]
    if kind == "graph":
        state["graph"].replay()
        return state["outputs"]
    if kind == "linear":
        return state["plan"].run(state["x"], state["w"], out_dtype=state["out"])
    if kind == "prefill":
        w = state["w"]
        if state["producer"] == "row":
            xq = ops.quantize_nvfp4_rowscale(state["x"])
        elif state["producer"] == "norm":
            xq = ops.rms_norm_quantize_nvfp4(state["x"], state["norm"], input_scale=w.input_scale)
        else:
            xq = ops.quantize_nvfp4(state["x"], w.input_scale)
        return state["plan"].run(xq, w, out_dtype=state["out"])
    if kind == "prefill_fp8":
        codes, scales = ops.quantize_fp8_dynamic(state["x"])
        weight, channel = state["w"]
        return state["plan"].run(codes, weight, scales, channel)
    if kind == "ffn":
        return state["ffn"].run(state["x"], state["residual"])
    return state["moe"].run(state["x"], state["logits"], state["gate_up"], state["down"], w_gate_up_interleaved=state["interleaved"])


# ---- the same results in 64 bits ----------------------------------------------------------------------------
def _nvfp4(v, scale):
    """What the NVFP4 codes of `v` stand for, without the global scale `scale`: the format's own 32-bit divisions (by the scale,
    the block maximum by 6, by the block scale) and roundings to nearest, ties to even; the result is exact in 32 bits."""
    out, rows = [], v.shape[0]
    scales = torch.as_tensor(scale, dtype=torch.float32, device="cuda").expand(rows, 1)
    six = torch.full((1,), 6.0, device="cuda")  # (divided by as a tensor: torch multiplies by the reciprocal of a number)
    for part, s in zip(v.float().split(4096), scales.split(4096)):
        q = (part / s).reshape(part.shape[0], -1, 16)
        block = (q.abs().amax(-1, keepdim=True) / six).clamp(max=448.0).to(torch.float8_e4m3fn).float()
        a = (q / torch.where(block == 0, 1.0, block)).abs()
        code = ((a > 0.25).float() + (a >= 0.75).float() + (a > 1.25).float() + (a >= 1.75).float()
                + 2 * (a > 2.5).float() + 2 * (a >= 3.5).float() + 4 * (a > 5.0).float())  # twice the value
        out.append((torch.copysign(0.5 * code, q) * block).reshape(part.shape))
    return torch.cat(out)


def _row_scale(x):
    """The smallest power of two that is no less than a row's largest value / (6 * 448)."""
    m, e = torch.frexp(x.double().abs().amax(1, keepdim=True) / 2688.0)
    return torch.ldexp(torch.ones_like(m), torch.where(m > 0.5, e, e - 1)).float()


def _fp8(x):
    scale = x.float().abs().amax(1, keepdim=True) / torch.full((1,), 448.0, device="cuda")
    return (x.float() / scale).to(torch.float8_e4m3fn).float(), scale.double()


def _nvfp4_normal(g, n, k, scale=None):
    """An NVFP4 weight of the cases: its values without, and its global scale."""
    w = _normal(g, (n, k), std=0.02)
    scale = (w.abs().max() / 2688.0) if scale is None else torch.tensor(scale, dtype=torch.float32, device="cuda")
    return _nvfp4(w, scale), scale.double()


def _times(x, w):
    """x . w^T in 64 bits, a slab of w at a time."""
    return torch.cat([x.double() @ part.double().t() for part in w.split(4096)], 1)


def _silu_mul(gate_up):
    gate, up = gate_up.double().chunk(2, -1)
    return gate / (1.0 + torch.exp(-gate)) * up


def exact(case, seed):
    """The results of `run` from the same inputs, products and sums in 64 bits; what the path stores in a narrower type between
    its steps (quantized operands, bf16 activations that the next layer reads) is rounded to that type here too."""
    g = _rng(seed)
    kind = case["kind"]
    if kind == "decode":
        t, h, i, dtype = case["tokens"], case["hidden"], case["inter"], _DTYPE[case["dtype"]]
        y, mid, out = _normal(g, (t, h), dtype), [], []
        for _ in range(case["layers"]):
            for results, n, k in ((mid, i, h), (out, h, i)):
                w, scale = _nvfp4_normal(g, n, k)
                results.append(_times(y, w) * scale)
                y = results[-1].to(dtype)
        return mid + out
    if kind == "decode_fp8":
        t, k, n = case["tokens"], case["k"], case["n"]
        outs, xs = [], [_normal(g, (t, k), torch.bfloat16) for _ in range(case["layers"])]
        for x in xs:
            (xq, s), (w, c) = _fp8(x), _fp8(_normal(g, (n, k), std=0.02))
            outs.append(_times(xq, w) * s * c.t())
        return outs
    if kind == "decode_moe":
        h, i, e, layers = case["hidden"], case["inter"], case["experts"], []
        for _ in range(case["layers"]):
            layers.append([[_nvfp4_normal(g, 2 * i, h, 0.1 / 2688.0) for _ in range(e)], [_nvfp4_normal(g, h, i, 0.1 / 2688.0) for _ in range(e)]])
        xs = [_normal(g, (h,)) for _ in layers]
        logits = [_normal(g, (e,)) for _ in layers]
        shared = [(_normal(g, (1,)), _normal(g, (h,))) for _ in layers]
        y, outs = _normal(g, (h,)), []
        for (gate_up, down), x, lg, (gate, sh) in zip(layers, xs, logits, shared):
            top, chosen = lg.double().topk(case["top_k"])
            total = y.double() + torch.sigmoid(gate.double()) * sh.double()
            for p, c in zip(torch.softmax(top, 0), chosen.tolist()):
                act = _silu_mul(_times(x[None], gate_up[c][0]) * gate_up[c][1])
                total = total + p * (_times(act, down[c][0]) * down[c][1])[0]
            outs.append(total)
            y = total.to(torch.bfloat16)
        return outs
    if kind == "linear":
        x = _normal(g, (case["tokens"], case["k"]), _DTYPE[case["dtype"]])
        w, scale = _nvfp4_normal(g, case["n"], case["k"])
        return _times(x, w) * scale
    if kind == "prefill":
        t, k, n = case["tokens"], case["k"], case["n"]
        x = _normal(g, (t, k), _DTYPE[case["dtype"]])
        w, scale = _nvfp4_normal(g, n, k)
        s = torch.tensor(4.5 / 2688.0, device="cuda")
        if case["producer"] == "row":
            s = _row_scale(x)
        elif case["producer"] == "norm":
            norm = _normal(g, (k,), std=0.1).add_(1.0).double()
            x = x.double() * torch.rsqrt(x.double().square().mean(1, keepdim=True) + 1e-6) * norm
        return _times(_nvfp4(x, s), w) * (scale * s.double())
    if kind == "prefill_fp8":
        (xq, s), (w, c) = _fp8(_normal(g, (case["tokens"], case["k"]), torch.bfloat16)), _fp8(_normal(g, (case["n"], case["k"]), std=0.02))
        return _times(xq, w) * s * c.t()
    if kind == "ffn":
        t, h, i = case["tokens"], case["hidden"], case["inter"]
        (gate_up, gu_scale), (down, dn_scale) = _nvfp4_normal(g, 2 * i, h), _nvfp4_normal(g, h, i)
        x, residual = _normal(g, (t, h), _DTYPE[case["dtype"]]), _normal(g, (t, h), torch.bfloat16)
        s, calibrated = _row_scale(x), torch.tensor(20.0 / 2688.0, device="cuda")
        act = _silu_mul(_times(_nvfp4(x, s), gate_up) * (gu_scale * s.double()))
        return _times(_nvfp4(act, calibrated), down) * (dn_scale * calibrated.double()) + residual.double()
    t, e, h, i = case["tokens"], case["experts"], case["hidden"], case["inter"]
    gate_up = [_nvfp4_normal(g, 2 * i, h, 0.1 / 2688.0) for _ in range(e)]
    down = [_nvfp4_normal(g, h, i, 0.1 / 2688.0) for _ in range(e)]
    x, logits = _normal(g, (t, h), _DTYPE[case["dtype"]]), _normal(g, (t, e))
    top, chosen = logits.double().topk(case["top_k"], 1)
    weights, xq, out = torch.softmax(top, 1), _nvfp4(x, 1.0), torch.zeros(t, h, dtype=torch.float64, device="cuda")
    for c in range(e):
        rows, slot = (chosen == c).nonzero(as_tuple=True)
        if len(rows):
            act = _silu_mul((_times(xq[rows], gate_up[c][0]) * gate_up[c][1]).to(torch.bfloat16))
            out[rows] += weights[rows, slot, None] * (_times(_nvfp4(act, 1.0), down[c][0]) * down[c][1])
    return out

def work(case):
    """Every input read once, every output written once; NVFP4 weights take 9/16 byte an element."""
    kind = case["kind"]
    size = {"bf16": 2, "f32": 4}
    if kind == "decode":
        t, h, i, b = case["tokens"], case["hidden"], case["inter"], size[case["dtype"]]
        return {"bytes": case["layers"] * (2 * h * i * 9 // 16 + t * (h + i) * b) + t * h * b, "flops": case["layers"] * 4 * t * h * i}
    if kind == "decode_fp8":
        t, k, n = case["tokens"], case["k"], case["n"]
        return {"bytes": case["layers"] * (n * k + 4 * n + 2 * t * (k + n)), "flops": case["layers"] * 2 * t * n * k}
    if kind == "decode_moe":
        h, i, s = case["hidden"], case["inter"], case["top_k"]
        return {"bytes": case["layers"] * (s * 3 * h * i * 9 // 16 + 4 * (3 * h + case["experts"])) + 4 * h, "flops": case["layers"] * s * 6 * h * i}
    if kind == "linear":
        t, k, n, b = case["tokens"], case["k"], case["n"], size[case["dtype"]]
        return {"bytes": n * k * 9 // 16 + t * (k + n) * b, "flops": 2 * t * n * k}
    if kind == "prefill":
        t, k, n = case["tokens"], case["k"], case["n"]
        return {"bytes": n * k * 9 // 16 + t * k * size[case["dtype"]] + t * n * size[case["out"]], "flops": 2 * t * n * k}
    if kind == "prefill_fp8":
        t, k, n = case["tokens"], case["k"], case["n"]
        return {"bytes": n * k + 4 * n + 2 * t * (k + n), "flops": 2 * t * n * k}
    if kind == "ffn":
        t, h, i = case["tokens"], case["hidden"], case["inter"]
        return {"bytes": 3 * h * i * 9 // 16 + t * h * (size[case["dtype"]] + 4), "flops": 6 * t * h * i}
    t, e, s, h, i = case["tokens"], case["experts"], case["top_k"], case["hidden"], case["inter"]
    touched = e * (1.0 - (1.0 - s / e) ** t)  # experts that some token chose
    return {"bytes": int(touched * 3 * h * i * 9 / 16) + t * (h * (size[case["dtype"]] + 4) + 4 * e), "flops": 6 * t * s * h * i}


def tolerance(case):
    """Against the same operands multiplied out in 64 bits and rounded to the output type: NVFP4 and FP8 products are summed
    almost exactly, so what differs is a last place of a bf16 result here and there (up to 0.008 of a value).  The decode
    linears expand bf16 activations into residual terms, which moves 4e-4 of a result and, through the chain of bf16 layers,
    5.5e-3 at its end."""
    kind, dtype = case["kind"], case.get("out", case.get("dtype"))
    if kind in ("decode", "linear", "prefill") and dtype == "f32":
        return {"rel": 1e-5}
    if kind == "decode":
        return {"rel": 0.01, "max": 0.09}
    if kind == "moe":  # the routes' down-projection rows are rounded to bf16 before they are weighted and summed
        return {"rel": 0.004, "max": 0.03}
    return {"rel": 0.002 if kind == "linear" else 0.001, "max": 0.03}
