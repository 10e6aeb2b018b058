"""The calls a program makes of this library, as cases to be timed: what a serving stack runs on quantized checkpoints.

Sizes are those of the benchmark (bench.py): the Llama-3.1-8B MLP (hidden 4096, intermediate 14336) and its
tensor-parallel shards, a hidden size of 5120 with 17408 columns for FP8 and NVFP4, the Qwen3-30B-A3B expert layer
(128 experts, top-8, hidden 2048, intermediate 768); row counts run from one token to a long prefill.

Decode-sized steps are what a serving loop replays from a CUDA graph: `graph` cases hold several layers of distinct
weights (more than the L2 holds where the layer is large enough), captured once over static buffers with workspaces that
the program keeps.  The other cases are eager calls of the modules and operators with their defaults, as a prefill step
or a plain torch program makes them.

    kind        one pass
    w4          one W4A16 linear (AWQ, GPTQ with or without act-order, compressed-tensors int4)
    mlp         [gate | up] + SwiGLU in one call, then the down projection, both W4A16
    moe         the routed expert layer on AWQ int4 experts: router, grouped expert FFN, combine
    fp8         FP8 W8A8 linears, per-channel weight scale, activations quantized per token inside the call
    fp8_block   FP8 W8A8 with 128 x 128 weight blocks, activations per token and per 128 of K
    nvfp4       NVFP4 W4A4 with a static activation scale
"""

from __future__ import annotations

import math

import torch

from emmy_b200 import linear, ops, ops_moe, ops_nvfp4

GROUP = 128
DTYPE = {"f16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # the smallest call: one 4096 x 4096 AWQ projection for one token, from a plain torch program
        {"name": "w4_awq_m1", "kind": "w4", "fmt": "awq", "order": "none", "rows": 1, "k": 4096, "n": 4096, "dtype": "f16", "graph": False, "layers": 1},
        # single-stream decode: four layers' MLPs for one token
        {"name": "mlp_m1", "kind": "mlp", "fmt": "gptq", "order": "blocks", "rows": 1, "k": 4096, "n": 14336, "dtype": "f16", "graph": True, "layers": 4},
        # a small decode batch, not a multiple of any tile
        {"name": "mlp_m12", "kind": "mlp", "fmt": "gptq", "order": "blocks", "rows": 12, "k": 4096, "n": 14336, "dtype": "bf16", "graph": True, "layers": 4},
        # a full decode batch
        {"name": "mlp_m64", "kind": "mlp", "fmt": "gptq", "order": "blocks", "rows": 64, "k": 4096, "n": 14336, "dtype": "f16", "graph": True, "layers": 3},
        # a short prompt or a chunk of one: ragged row count
        {"name": "mlp_m300", "kind": "mlp", "fmt": "awq", "order": "none", "rows": 300, "k": 4096, "n": 14336, "dtype": "bf16", "graph": False, "layers": 1},
        # a long prefill
        {"name": "mlp_m4096", "kind": "mlp", "fmt": "gptq", "order": "blocks", "rows": 4096, "k": 4096, "n": 14336, "dtype": "f16", "graph": False, "layers": 1},
        # the expert layer: one token, a decode batch, a prefill
        {"name": "moe_t1", "kind": "moe", "rows": 1, "experts": 128, "topk": 8, "k": 2048, "n": 768, "dtype": "bf16", "graph": True, "layers": 4},
        {"name": "moe_t64", "kind": "moe", "rows": 64, "experts": 128, "topk": 8, "k": 2048, "n": 768, "dtype": "bf16", "graph": True, "layers": 2},
        {"name": "moe_t4096", "kind": "moe", "rows": 4096, "experts": 128, "topk": 8, "k": 2048, "n": 768, "dtype": "bf16", "graph": False, "layers": 1},
        # FP8 decode batch: the wide projection of four layers
        {"name": "fp8_m32", "kind": "fp8", "rows": 32, "k": 5120, "n": 17408, "dtype": "bf16", "graph": True, "layers": 4},
        # block-scaled FP8 prefill
        {"name": "fp8_block_m2048", "kind": "fp8_block", "rows": 2048, "k": 5120, "n": 17408, "dtype": "bf16", "graph": False, "layers": 1},
        # NVFP4 prefill
        {"name": "nvfp4_m4096", "kind": "nvfp4", "rows": 4096, "k": 5120, "n": 17408, "dtype": "bf16", "graph": False, "layers": 1},
    ]


def _rows(rng, most):
    """Row counts spread over their logarithm; one in three a power of two (batch sizes), the rest whatever comes."""
    r = math.exp(rng.uniform(0.0, math.log(most)))
    return min(most, 1 << round(math.log2(r))) if rng.random() < 1 / 3 else max(1, min(most, round(r)))


def draw(rng):
    kind = rng.choice(["w4", "w4", "w4", "mlp", "mlp", "mlp", "moe", "moe", "fp8", "fp8", "fp8_block", "nvfp4", "nvfp4"])
    dtype = rng.choice(["f16", "bf16"])
    case = {"kind": kind, "dtype": dtype}
    if kind in ("w4", "mlp"):
        fmt, order = rng.choice([("awq", "none"), ("gptq", "none"), ("gptq", "blocks"), ("gptq", "scattered"), ("ct", "none")])
        if kind == "mlp" and order == "scattered":
            order = "blocks"  # the fused [gate | up] call above 16 rows takes weights without a row permutation
        tp = rng.choice([1, 1, 2, 4, 8])
        case.update(fmt=fmt, order=order, rows=_rows(rng, 4096))
        if kind == "mlp":
            hidden, inter = rng.choice([(4096, 14336), (5120, 17408)])
            case.update(k=hidden, n=inter // tp)
        else:
            # projections of a decoder layer and their shards, and one with an odd width
            k, n = rng.choice([(4096, 4096), (4096, 6144), (4096, 14336 // tp), (14336 // tp, 4096), (5120, 17408 // tp), (5120, 16 * rng.randint(65, 900))])
            case.update(k=k, n=n)
    elif kind == "moe":
        experts, topk = rng.choice([(128, 8), (128, 8), (64, 6), (32, 4)])
        k, n = rng.choice([(2048, 768), (2048, 768), (2048, 1024), (1024, 512)])
        case.update(rows=_rows(rng, 4096), experts=experts, topk=topk, k=k, n=n)
    else:
        step = {"fp8": 16, "fp8_block": 128, "nvfp4": 8}[kind]
        k, n = rng.choice([(5120, 17408), (5120, 5120), (4096, 6144), (5120, step * rng.randint(1024 // step, 16384 // step))])
        case.update(rows=_rows(rng, 8192), k=k, n=n)
    # decode steps are graph replays over a few layers, everything larger an eager call; one small call in four is eager too
    case["graph"] = case["rows"] <= 64 and rng.random() < 0.75
    case["layers"] = rng.choice([2, 3, 4]) if case["graph"] else 1
    return case


# ------------------------------------------------------------------------------------------------------------- inputs


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + 7919 * salt) % (1 << 62))


def _words(gen, *shape):
    return torch.randint(-(2**31), 2**31 - 1, shape, dtype=torch.int32, device="cuda", generator=gen)


def _scales(gen, dtype, *shape):
    return (torch.rand(shape, device="cuda", generator=gen) * (2e-2 - 1e-3) + 1e-3).to(dtype)


def _w4_tensors(gen, fmt, order, k, n, lead=()):
    """A checkpoint's tensors: int4 uniform, zero points uniform (AWQ, compressed-tensors) or the symmetric 8 (GPTQ)."""
    qweight = _words(gen, *lead, k, n // 8) if fmt == "awq" else _words(gen, *lead, k // 8, n)
    if fmt == "gptq":
        qzeros = torch.full((*lead, k // GROUP, n // 8), 0x77777777, dtype=torch.int32, device="cuda")
    else:
        qzeros = _words(gen, *lead, k // GROUP, n // 8)
    scales = _scales(gen, torch.bfloat16 if fmt == "ct" else torch.float16, *lead, k // GROUP, n)
    g_idx = None
    if order == "blocks":
        g_idx = torch.randperm(k // GROUP, device="cuda", generator=gen)[torch.arange(k, device="cuda") // GROUP].int()
    elif order == "scattered":
        g_idx = (torch.randperm(k, device="cuda", generator=gen) // GROUP).int()
    return qweight, qzeros, scales, g_idx


def _w4_weight(gen, fmt, order, k, n):
    qweight, qzeros, scales, g_idx = _w4_tensors(gen, fmt, order, k, n)
    return ops.w4_repack(qweight, qzeros, scales, GROUP, fmt, g_idx=g_idx)


def _zeros(nbytes):
    return torch.zeros(nbytes + 256, dtype=torch.uint8, device="cuda")


def _layers_w4(case, seed):
    m, k, n, layers, dtype = case["rows"], case["k"], case["n"], case["layers"], DTYPE[case["dtype"]]
    x = torch.randn(m, k, device="cuda", generator=_gen(seed)).to(dtype)
    if not case["graph"]:
        qweight, qzeros, scales, g_idx = _w4_tensors(_gen(seed, 1), case["fmt"], case["order"], k, n)
        layer = linear.W4A16Linear(k, n, GROUP, case["fmt"], act_order=g_idx is not None, scale_dtype=scales.dtype)
        layer.qweight, layer.qzeros, layer.scales = qweight, qzeros, scales
        if g_idx is not None:
            layer.g_idx = g_idx
        layer.finalize()
        return lambda: [layer(x)]
    weights = [_w4_weight(_gen(seed, 1 + i), case["fmt"], case["order"], k, n) for i in range(layers)]
    ws = _zeros(ops.L.load().eq_w4a16_workspace_bytes(m, n, k))
    outs = [torch.empty(m, n, dtype=dtype, device="cuda") for _ in weights]
    return lambda: [ops.w4a16_linear(x, w, workspace=ws, out=y) for w, y in zip(weights, outs)]


def _layers_mlp(case, seed):
    m, k, n, layers, dtype = case["rows"], case["k"], case["n"], case["layers"], DTYPE[case["dtype"]]
    x = torch.randn(m, k, device="cuda", generator=_gen(seed)).to(dtype)
    fmt, order = case["fmt"], case["order"]
    gate_up = [ops.w4_concat([_w4_weight(_gen(seed, 10 * i + j), fmt, order, k, n) for j in (1, 2)]) for i in range(layers)]
    down = [_w4_weight(_gen(seed, 10 * i + 3), fmt, "none", n, k) for i in range(layers)]
    if not case["graph"]:
        return lambda: [ops.w4a16_linear(ops.w4a16_gate_up_swiglu(x, g), d) for g, d in zip(gate_up, down)]
    lib = ops.L.load()
    ws_gu, ws_dn = _zeros(lib.eq_w4a16_gate_up_workspace_bytes(m, n, k)), _zeros(lib.eq_w4a16_workspace_bytes(m, k, n))
    hidden = torch.empty(m, n, dtype=dtype, device="cuda")
    outs = [torch.empty(m, k, dtype=dtype, device="cuda") for _ in down]

    def step():
        for g, d, y in zip(gate_up, down, outs):
            ops.w4a16_gate_up_swiglu(x, g, workspace=ws_gu, out=hidden)
            ops.w4a16_linear(hidden, d, workspace=ws_dn, out=y)
        return outs

    return step


def _layers_moe(case, seed):
    t, e, k, n, dtype = case["rows"], case["experts"], case["k"], case["n"], DTYPE[case["dtype"]]
    topk = case["topk"]
    x = torch.randn(t, k, device="cuda", generator=_gen(seed)).to(dtype)
    logits = torch.randn(t, e, device="cuda", generator=_gen(seed, 1))

    def stacks(i):
        return [_w4_tensors(_gen(seed, 10 * i + 2 + j), "awq", "none", *shape, lead=(e,))[:3] for j, shape in enumerate([(k, 2 * n), (n, k)])]

    if not case["graph"]:
        layer = linear.QuantMoE(topk).load_experts(*stacks(0), GROUP, "awq")
        return lambda: [layer(x, logits)]
    weights = [ops_moe.moe_repack(*stacks(i), GROUP, "awq") for i in range(case["layers"])]
    ws = ops_moe.moe_workspace(t, weights[0], topk, x.device)
    outs = [torch.empty(t, k, dtype=dtype, device="cuda") for _ in weights]
    return lambda: [ops_moe.moe_forward(x, logits, w, topk, workspace=ws, out=y) for w, y in zip(weights, outs)]


def _layers_fp8(case, seed):
    m, k, n, layers, dtype = case["rows"], case["k"], case["n"], case["layers"], DTYPE[case["dtype"]]
    x = torch.randn(m, k, device="cuda", generator=_gen(seed)).to(dtype)
    weights = []
    for i in range(layers):
        w = torch.randn(n, k, device="cuda", generator=_gen(seed, 1 + i)) * 0.02
        bits, scale = ops.quant_fp8_per_token(w)  # the per-channel rule is the per-token rule on the weight's rows
        weights.append((bits, scale.reshape(-1).contiguous()))
    if not case["graph"]:
        layer = linear.FP8Linear(k, n)
        layer.weight, layer.weight_scale = weights[0]
        return lambda: [layer(x)]
    ws = ops.fp8_workspace(m, k, x.device)
    outs = [torch.empty(m, n, dtype=dtype, device="cuda") for _ in weights]
    return lambda: [ops.fp8_linear(x, b, s, workspace=ws, out=y) for (b, s), y in zip(weights, outs)]


def _layers_fp8_block(case, seed):
    m, k, n, layers, dtype = case["rows"], case["k"], case["n"], case["layers"], DTYPE[case["dtype"]]
    x = torch.randn(m, k, device="cuda", generator=_gen(seed)).to(dtype)
    weights = []
    for i in range(layers):
        blocks = (torch.randn(n, k, device="cuda", generator=_gen(seed, 1 + i)) * 0.02).reshape(n // 128, 128, k // 128, 128)
        s = (blocks.abs().amax(dim=(1, 3)).clamp_min(1e-12) / 448.0).float()
        bits = (blocks / s[:, None, :, None]).reshape(n, k).to(torch.float8_e4m3fn).view(torch.uint8)
        weights.append((bits.contiguous(), s.contiguous()))
    if not case["graph"]:
        layer = linear.FP8BlockLinear(k, n)
        layer.weight, layer.weight_scale_inv = weights[0]
        return lambda: [layer(x)]
    ws = _zeros(ops.L.load().eq_fp8_block_workspace_bytes(m, k))
    outs = [torch.empty(m, n, dtype=dtype, device="cuda") for _ in weights]
    return lambda: [ops.fp8_block_linear(x, b, s, workspace=ws, out=y) for (b, s), y in zip(weights, outs)]


def _layers_nvfp4(case, seed):
    m, k, n, layers, dtype = case["rows"], case["k"], case["n"], case["layers"], DTYPE[case["dtype"]]
    x = torch.randn(m, k, device="cuda", generator=_gen(seed)).to(dtype)
    input_scale = ops_nvfp4.nvfp4_global_scale(x)
    weights = [ops_nvfp4.quant_nvfp4_weight(torch.randn(n, k, device="cuda", generator=_gen(seed, 1 + i)) * 0.02) for i in range(layers)]
    if not case["graph"]:
        layer = linear.NVFP4Linear(k, n)
        (layer.weight, layer.weight_scale, layer.weight_scale_2), layer.input_scale = weights[0], input_scale
        layer.finalize()
        return lambda: [layer(x)]
    tiled = [(p, ops_nvfp4.nvfp4_tile_weight_scales(sf, k), s2) for p, sf, s2 in weights]
    ws = ops_nvfp4.nvfp4_workspace(m, k, x.device)
    outs = [torch.empty(m, n, dtype=dtype, device="cuda") for _ in tiled]
    return lambda: [ops_nvfp4.nvfp4_linear(x, p, sf, s2, input_scale, workspace=ws, out=y) for (p, sf, s2), y in zip(tiled, outs)]


_BUILD = {"w4": _layers_w4, "mlp": _layers_mlp, "moe": _layers_moe, "fp8": _layers_fp8, "fp8_block": _layers_fp8_block, "nvfp4": _layers_nvfp4}


def prepare(case, seed):
    with torch.no_grad():
        step = _BUILD[case["kind"]](case, seed)
        if not case["graph"]:
            return {"step": step}
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            step()
        torch.cuda.current_stream().wait_stream(stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = step()
    return {"step": step, "graph": graph, "outs": outs}


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["outs"]
    with torch.no_grad():
        return state["step"]()


# --------------------------------------------------------------------------------------------- the same in 64 bits


def _nibbles(words, fmt, along_rows):
    shifts = (0, 16, 4, 20, 8, 24, 12, 28) if fmt == "awq" else (0, 4, 8, 12, 16, 20, 24, 28)
    parts = [(words >> s) & 15 for s in shifts]
    if along_rows:
        return torch.stack(parts, dim=1).reshape(8 * words.shape[0], words.shape[1])
    return torch.stack(parts, dim=2).reshape(words.shape[0], 8 * words.shape[1])


def _w4_values(fmt, qweight, qzeros, scales, g_idx=None):
    """Checkpoint tensors of one linear -> its weight [K, N], 64 bits."""
    q = _nibbles(qweight, fmt, fmt != "awq").double()
    z = _nibbles(qzeros, fmt, False).double() + (1.0 if fmt == "gptq" else 0.0)
    g = (torch.arange(q.shape[0], device=q.device) // GROUP) if g_idx is None else g_idx.long()
    return (q - z[g]) * scales.double()[g]


def _swiglu(gate_up):
    gate, up = gate_up.chunk(2, dim=-1)
    return torch.nn.functional.silu(gate) * up


def _fp8_codes(v, amax):
    """v / (max(amax, 1e-12) / 448) in f32, rounded to e4m3: (the codes' values, the scales), 64 bits."""
    s = amax.clamp_min(1e-12) / 448.0
    return (v / s).to(torch.float8_e4m3fn).double(), s.double()


def _e2m1(v):
    a = v.abs()
    pitch = torch.where(a < 2, 0.5, torch.where(a < 4, 1.0, 2.0))
    return torch.copysign((torch.round(a / pitch) * pitch).clamp_max(6.0), v).double()


def _nvfp4_activation(x):
    """The static rule: block scales relative to the global one, codes of x / (scale * global), every step in f32."""
    s2 = x.abs().amax().clamp_min(1e-12) / (6.0 * 448.0)
    blocks = x.reshape(x.shape[0], -1, 16)
    sixth = torch.ones((), device=x.device) / 6.0
    bits = (blocks.abs().amax(dim=-1) * sixth * (1.0 / s2)).clamp_max(448.0).to(torch.float8_e4m3fn).float()
    codes = _e2m1(blocks / (bits * s2).clamp_min(1e-12)[..., None])
    return (codes * bits.double()[..., None]).reshape(x.shape) * s2.double()


def _nvfp4_weight(w):
    """The weight rule: block scale = block amax / 6 as e4m3 relative to scale_2, codes of w / f16(scale * scale_2)."""
    s2 = w.abs().amax().clamp_min(1e-12) / (6.0 * 448.0)
    blocks = w.reshape(w.shape[0], -1, 16)
    bits = (blocks.abs().amax(dim=-1) / 6.0 / s2).clamp_max(448.0).to(torch.float8_e4m3fn).float()
    fused = (bits * s2).half().float()[..., None]
    codes = _e2m1(torch.where(fused != 0, blocks / fused, torch.zeros_like(blocks)))
    return (codes * bits.double()[..., None]).reshape(w.shape) * s2.double()


def exact(case, seed):
    """run()'s outputs from the same checkpoint tensors and the same activation codes, everything after them in 64 bits."""
    with torch.no_grad():
        m, k, n, kind, dtype = case["rows"], case["k"], case["n"], case["kind"], DTYPE[case["dtype"]]
        x = torch.randn(m, k, device="cuda", generator=_gen(seed)).to(dtype)
        outs = []
        for i in range(case["layers"]):
            if kind == "w4":
                outs.append(x.double() @ _w4_values(case["fmt"], *_w4_tensors(_gen(seed, 1 + i), case["fmt"], case["order"], k, n)))
            elif kind == "mlp":
                fmt, order = case["fmt"], case["order"]
                gate, up = (x.double() @ _w4_values(fmt, *_w4_tensors(_gen(seed, 10 * i + j), fmt, order, k, n)) for j in (1, 2))
                hidden = torch.nn.functional.silu(gate) * up
                outs.append(hidden @ _w4_values(fmt, *_w4_tensors(_gen(seed, 10 * i + 3), fmt, "none", n, k)))
            elif kind == "moe":
                e, topk = case["experts"], case["topk"]
                logits = torch.randn(m, e, device="cuda", generator=_gen(seed, 1)).double()
                scores, ids = torch.softmax(logits, dim=-1).topk(topk, dim=-1)
                scores = scores / scores.sum(dim=-1, keepdim=True)
                gate_up, down = (_w4_tensors(_gen(seed, 10 * i + 2 + j), "awq", "none", *s, lead=(e,))[:3] for j, s in enumerate([(k, 2 * n), (n, k)]))
                y = torch.zeros(m, k, dtype=torch.float64, device="cuda")
                for j in range(e):
                    rows, slot = (ids == j).nonzero(as_tuple=True)
                    if rows.numel():
                        h = _swiglu(x[rows].double() @ _w4_values("awq", *(t[j] for t in gate_up)))
                        y.index_add_(0, rows, scores[rows, slot, None] * (h @ _w4_values("awq", *(t[j] for t in down))))
                outs.append(y)
            else:
                w = torch.randn(n, k, device="cuda", generator=_gen(seed, 1 + i)) * 0.02
                xf = x.float()
                if kind == "fp8":
                    (xq, xs), (wq, wscale) = (_fp8_codes(v, v.abs().amax(dim=1, keepdim=True)) for v in (xf, w))
                    outs.append((xq @ wq.T) * xs * wscale.reshape(1, -1))
                elif kind == "fp8_block":
                    xb = xf.reshape(m, k // 128, 128)
                    xq, xs = _fp8_codes(xb, xb.abs().amax(dim=2, keepdim=True))
                    blocks = w.reshape(n // 128, 128, k // 128, 128)
                    s = blocks.abs().amax(dim=(1, 3)).clamp_min(1e-12) / 448.0
                    bits = (blocks / s[:, None, :, None]).to(torch.float8_e4m3fn).double()
                    outs.append((xq * xs).reshape(m, k) @ (bits * s.double()[:, None, :, None]).reshape(n, k).T)
                else:
                    outs.append(_nvfp4_activation(xf) @ _nvfp4_weight(w).T)
        return outs


# -------------------------------------------------------------------------------------------------- bytes and flops


def _w4_bytes(k, n):
    return k * n / 2 + (k // GROUP) * (n / 2 + 2 * n)  # nibbles, zero points, 16-bit scales


def work(case):
    m, k, n, kind = case["rows"], case["k"], case["n"], case["kind"]
    io = 2 * m * k + 2 * m * n
    if kind == "w4":
        b, f = _w4_bytes(k, n) + io, 2.0 * m * k * n
    elif kind == "mlp":
        b, f = _w4_bytes(k, 2 * n) + _w4_bytes(n, k) + 4 * m * k, 6.0 * m * k * n
    elif kind == "moe":
        e, topk = case["experts"], case["topk"]
        hit = e * (1.0 - (1.0 - topk / e) ** m)  # experts that m tokens touch, on average
        b, f = hit * (_w4_bytes(k, 2 * n) + _w4_bytes(n, k)) + 4 * m * k + 4 * m * e, 6.0 * m * topk * k * n
    elif kind == "fp8":
        b, f = k * n + 4 * n + io, 2.0 * m * k * n
    elif kind == "fp8_block":
        b, f = k * n + (k // 128) * (n // 128) * 4 + io, 2.0 * m * k * n
    else:
        b, f = k * n / 2 + k * n / 16 + 8 + io, 2.0 * m * k * n
    return {"bytes": case["layers"] * b, "flops": case["layers"] * f}


def tolerance(case):
    """Outputs are rounded to the activation dtype; a W4 kernel may apply the group scale to the weight (one more rounding
    per weight, two where the scale is stored in the other 16-bit type) or to the sums, and an MLP rounds its intermediate
    as well.  Against a 64-bit evaluation of either form the paths measure, f16 | bf16: linear 2.9e-4 | 3.1e-3, MLP
    5.6e-4 | 5.8e-3.  FP8 and NVFP4 codes are the same everywhere, so only the order of the f32 sums and the output's
    rounding (2.1e-4 | 1.7e-3) remain."""
    f16 = case["dtype"] == "f16"
    if case["kind"] in ("fp8", "fp8_block", "nvfp4"):
        return {"rel": 8e-4 if f16 else 6e-3}
    if case["kind"] == "w4":
        return {"rel": 1.2e-3 if f16 else 1.2e-2}
    return {"rel": 2.2e-3 if f16 else 2e-2}
