"""The work whose speed is measured: what programs built on this package have it do, over the sizes they use.

Sizes are those of the repository's benchmark and tests -- Llama-3.1-8B shapes, the recipes' own block sizes and
formats -- with ragged token counts, short batches and odd extents beside the round ones.  Each kind below is one
recipe's path through the public entry points:

* ``mx_linear``: a converted microscaling graph's linear site -- ``quantize_mx`` of the activation, then
  ``linear_mx`` with a weight that was quantized when the graph was converted.  ``int8`` (blocks of 16, power-of-two
  scales) and ``nf4`` (``lut4_to_int6``, blocks of 64, fp8_e5m3 scales), from a handful of rows to a prefill.
* ``fp8_layer`` / ``nvfp4_layer``: a prefill through one decoder layer of the FP8 and the NVFP4 recipe.
* ``decode``: one decode step of an MXNF4 decoder layer over a 2-bit KIVI cache, served the way a decode loop is:
  a captured step is replayed on the new token's hidden states.
* ``kivi``: the cache written after a prefill (keys grouped along the positions, values along the channels) and
  read back, as a prompt that attends to its own quantized cache needs both.
* ``gptq``: one linear of a calibration run: the Hessian of a chunk of activations, then the solve.
* ``fp8_train`` / ``nvfp4_train``: a training step's forward and backward of one linear in real FP8 (with the
  backward of the norm in front of it) and in NVFP4 (rotated, stochastically rounded gradients).
"""

import math

import torch

import voyager_b200 as vb

W = vb.workloads
SHAPE = W.LLAMA_8B
Q = torch.ops.quantized_ops
G = torch.ops.voyager_gpu

# element table, block, quant_max, power-of-two scales, scale table
MX_FORMATS = {"int8": ("int8", 16, 127.0, True, None), "nf4": ("lut4_to_int6", 64, 31.0, False, "fp8_e5m3")}


def listed():
    return [
        # a few rows against one projection: a short decode batch in a graph that keeps the operator's own storage
        {"name": "mx_int8_rows7", "kind": "mx_linear", "format": "int8", "tokens": 7, "n": 4096, "k": 4096},
        # the repository's MXINT8 linear
        {"name": "mx_int8_2048", "kind": "mx_linear", "format": "int8", "tokens": 2048, "n": 4096, "k": 4096},
        # a prompt of no round length through the up projection in the lookup-format recipe
        {"name": "mx_nf4_1000", "kind": "mx_linear", "format": "nf4", "tokens": 1000, "n": 14336, "k": 4096},
        # the repository's headline layer, and a prompt that fills no tile
        {"name": "fp8_layer_2048", "kind": "fp8_layer", "tokens": 2048},
        {"name": "fp8_layer_776", "kind": "fp8_layer", "tokens": 776},
        # the long prefill of the NVFP4 model, one of its layers
        {"name": "nvfp4_layer_8192", "kind": "nvfp4_layer", "tokens": 8192},
        # the decode step at the benchmark's batch and context, and a single short conversation
        {"name": "decode_b16_4096", "kind": "decode", "batch": 16, "cached": 3968, "recent": 128},
        {"name": "decode_b1_1013", "kind": "decode", "batch": 1, "cached": 960, "recent": 53},
        # four prompts' caches
        {"name": "kivi_b4_3968", "kind": "kivi", "batch": 4, "positions": 3968},
        # one attention projection of a calibration run
        {"name": "gptq_4096", "kind": "gptq", "n": 4096, "k": 4096, "tokens": 16384},
        # forward and backward of one linear
        {"name": "fp8_train_4096", "kind": "fp8_train", "tokens": 4096, "n": 4096, "k": 4096},
        {"name": "nvfp4_train_4096", "kind": "nvfp4_train", "tokens": 4096, "n": 4096, "k": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("mx_linear", "fp8_layer", "nvfp4_layer", "decode", "kivi", "gptq", "fp8_train", "nvfp4_train"))
    case = {"kind": kind}
    if kind == "mx_linear":
        n = _log(rng, 512, 14336)
        case.update(format=rng.choice(("int8", "nf4")), tokens=_log(rng, 1, 4096), n=n if rng.random() < 0.25 else -(-n // 8) * 8,
                    k=64 * _log(rng, 8, 128))
    elif kind == "fp8_layer":
        t = _log(rng, 64, 2048)
        # the layer takes prompts padded to a multiple of 8
        case.update(tokens=-(-t // 8) * 8 if rng.random() < 0.5 else max(128, t // 128 * 128))
    elif kind == "nvfp4_layer":
        t = _log(rng, 128, 8192)
        case.update(tokens=min(t, 3000) if rng.random() < 0.5 else t // 128 * 128)
    elif kind == "decode":
        case.update(batch=rng.randint(1, 16), cached=64 * _log(rng, 4, 62), recent=rng.randint(17, 128))
    elif kind == "kivi":
        case.update(batch=rng.randint(1, 4), positions=64 * _log(rng, 4, 62))
    elif kind == "gptq":
        case.update(n=8 * _log(rng, 64, 512), k=128 * _log(rng, 4, 32), tokens=_log(rng, 2048, 16384))
    elif kind == "fp8_train":
        case.update(tokens=_log(rng, 128, 4096), n=16 * _log(rng, 32, 256), k=16 * _log(rng, 32, 256))
    else:
        case.update(tokens=64 * _log(rng, 2, 64), n=64 * _log(rng, 8, 64), k=64 * _log(rng, 8, 64))
    return case


# ---------------------------------------------------------------------------
# what a program holds before the call
# ---------------------------------------------------------------------------
def _randn(seed, *dims, std=1.0, outliers=False):
    """N(0, std) in bfloat16; activations carry 0.1 % of entries at twenty times the rest."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(*dims, generator=g, device="cuda") * std
    if outliers:
        x = torch.where(torch.rand(dims, generator=g, device="cuda") < 0.001, x * 20, x)
    return x.bfloat16()


def _mx_tables(fmt):
    name, block, quant_max, pow2, scale_name = MX_FORMATS[fmt]
    table = vb.get_quantization_map(name, "cuda")
    scale_table = None if scale_name is None else vb.get_quantization_map(scale_name, "cuda")
    if fmt == "nf4":
        index, levels = vb.formats.index_table(table)
        return index, block, quant_max, pow2, scale_table, levels
    return table, block, quant_max, pow2, scale_table, None


def _prepare_mx_linear(case, seed):
    table, block, quant_max, pow2, scale_table, levels = _mx_tables(case["format"])
    mid = None if levels is None else (levels[:-1] + levels[1:]) / 2
    args = (table, [-1], block, quant_max, pow2, scale_table, mid)
    ws, wc = Q.quantize_mx(_randn(2 * seed, case["n"], case["k"], std=0.02), *args)
    return {"x": _randn(2 * seed + 1, case["tokens"], case["k"], outliers=True), "args": args, "ws": ws, "wc": wc,
            "block": block, "levels": levels}


def _run_mx_linear(s):
    scale, codes = Q.quantize_mx(s["x"], *s["args"])
    return Q.linear_mx(codes, s["wc"], None, input_scale=scale, weight_scale=s["ws"], block_size=s["block"],
                       input_code=s["levels"], weight_code=s["levels"])


def _prepare_fp8_layer(case, seed):
    params = W.make_layer_params_on_device(2 * seed, SHAPE, "cuda")
    # scales from a calibration prompt of its own
    scales = W.calibrate_fp8_scales(_randn(2 * seed + 7, 256, SHAPE.hidden), params, SHAPE)
    return {"layer": W.Fp8DecoderLayer(params, scales, SHAPE), "x": _randn(2 * seed + 1, case["tokens"], SHAPE.hidden)}


def _prepare_nvfp4_layer(case, seed):
    params = W.make_layer_params_on_device(2 * seed, SHAPE, "cuda")
    return {"layer": W.Nvfp4DecoderLayer(params, SHAPE), "x": _randn(2 * seed + 1, case["tokens"], SHAPE.hidden)}


def _run_layer(s):
    return s["layer"](s["x"])


def _prepare_decode(case, seed):
    t, sh, b = W.nf4_tables("cuda"), SHAPE, case["batch"]
    rows = {"qkv": ((sh.heads + 2 * sh.kv_heads) * sh.head_dim, sh.hidden), "o": (sh.hidden, sh.heads * sh.head_dim),
            "gate_up": (2 * sh.intermediate, sh.hidden), "down": (sh.hidden, sh.intermediate)}
    weights = {}
    for i, (name, (n, k)) in enumerate(rows.items()):
        scale, codes = Q.quantize_mx(_randn(16 * seed + i, n, k, std=0.02), t["index"], [-1], 64, 31.0, False, t["e5m3"], t["mid"])
        weights[name] = vb.packed.pack_lut4_weight(codes, scale, t["levels"], 64, check=False)
    weights["ln1"] = weights["ln2"] = torch.ones(sh.hidden, dtype=torch.bfloat16, device="cuda")

    def kv(i, positions):
        return _randn(16 * seed + 4 + i, b, sh.kv_heads, positions, sh.head_dim)

    cache = {"k": vb.kivi.quantize_cache(kv(0, case["cached"]), t["uint2"], -2, 64, 2, t["e4m3"]),
             "v": vb.kivi.quantize_cache(kv(1, case["cached"]), t["uint2"], -1, 64, 2, t["e4m3"]),
             "k_res": kv(2, case["recent"]), "v_res": kv(3, case["recent"])}
    # the residual stream lies within +-8
    layer = W.Mxnf4DecodeLayer(weights, t, cache, torch.tensor(8.0 / 448.0, dtype=torch.bfloat16, device="cuda"), sh)
    cos, sin = W.rope_tables(case["cached"] + case["recent"], sh, "cuda")
    rope = (cos[-1].contiguous(), sin[-1].contiguous())
    x = _randn(16 * seed + 8, b, sh.hidden)
    # a decode loop captures its step once and replays it for every token
    static = x.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        layer(static, rope)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = layer(static, rope)
    return {"x": x, "static": static, "graph": graph, "out": out, "cache": cache, "layer": layer, "rope": rope}


def _run_decode(s):
    s["static"].copy_(s["x"])
    s["graph"].replay()
    # the token's keys and values take the last slot of the recent window
    return s["out"], s["cache"]["k_res"], s["cache"]["v_res"]


def _prepare_kivi(case, seed):
    dims = (case["batch"], SHAPE.kv_heads, case["positions"], SHAPE.head_dim)
    return {"k": _randn(2 * seed, *dims), "v": _randn(2 * seed + 1, *dims),
            "uint2": vb.get_quantization_map("uint2", "cuda"), "e4m3": vb.get_quantization_map("fp8_e4m3", "cuda")}


def _run_kivi(s):
    k = vb.kivi.quantize_cache(s["k"], s["uint2"], -2, 64, 2, s["e4m3"])
    v = vb.kivi.quantize_cache(s["v"], s["uint2"], -1, 64, 2, s["e4m3"])
    return [k.packed, k.scale, k.zero_point, v.packed, v.scale, v.zero_point, k.read(), v.read()]


def _prepare_gptq(case, seed):
    k, tokens = case["k"], case["tokens"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    # calibration rows: independent normals with a rank-64 correlated part
    low = torch.randn(tokens, 64, generator=g, device="cuda") @ torch.randn(64, k, generator=g, device="cuda")
    x = (0.7 * torch.randn(tokens, k, generator=g, device="cuda") + 0.3 * low / 8).bfloat16()
    return {"x": x, "w": _randn(seed + 1, case["n"], k, std=0.02), "qmap": vb.get_quantization_map("uint4", "cuda")}


def _run_gptq(s):
    h = vb.gptq.accumulate_hessian(None, s["x"])
    return vb.gptq.compensate_weight_affine(s["w"], h, s["x"].shape[0], s["qmap"], 0.0, 15.0, 128, 0.01)


def _prepare_fp8_train(case, seed):
    m, n, k = case["tokens"], case["n"], case["k"]
    x, w, g = _randn(8 * seed, m, k), _randn(8 * seed + 1, n, k, std=0.02), _randn(8 * seed + 2, m, n, std=1e-3)
    # delayed scaling: the scales are there before the step
    scales = {name: (t.abs().amax() / 448.0).float() for name, t in (("x", x), ("w", w), ("g", g))}
    h = _randn(8 * seed + 3, m, k)
    return {"x": x, "w": w, "g": g, "h": h, "residual": _randn(8 * seed + 4, m, k, std=1e-3),
            "rsqrt": torch.rsqrt(h.float().pow(2).mean(-1, keepdim=True) + 1e-5), "gain": _randn(8 * seed + 5, k),
            "sx": scales["x"], "sw": scales["w"], "sg": scales["g"], "y_scale": scales["x"] * scales["w"],
            "dx_scale": scales["g"] * scales["w"], "dw_scale": scales["g"] * scales["x"]}


def _run_fp8_train(s):
    e4m3 = torch.float8_e4m3fn
    x8, xt8, x_amax = G.cast_transpose_fp8(s["x"], s["sx"], e4m3)
    w8, wt8, w_amax = G.cast_transpose_fp8(s["w"], s["sw"], e4m3)
    y = vb.fp8.fp8_linear(x8, w8, s["y_scale"])
    g8, gt8, g_amax = G.cast_transpose_fp8(s["g"], s["sg"], e4m3)
    dx = vb.fp8.fp8_linear(g8, wt8, s["dx_scale"])
    dw = vb.fp8.fp8_linear(gt8, xt8, s["dw_scale"])
    dh, dgain = vb.training.rmsnorm_backward([dx], s["h"], s["rsqrt"], s["gain"], s["residual"])
    return y, dw, dh, dgain, x_amax, w_amax, g_amax


def _prepare_nvfp4_train(case, seed):
    m, n, k = case["tokens"], case["n"], case["k"]
    return {"x": _randn(4 * seed, m, k), "w": _randn(4 * seed + 1, n, k, std=0.02), "g": _randn(4 * seed + 2, m, n, std=1e-3),
            "hadamard": vb.ops.hadamard_matrix("cuda"), "one": torch.ones((), device="cuda"),
            "seeds": [torch.tensor(2 * seed + i, dtype=torch.int64, device="cuda") for i in range(2)]}


def _run_nvfp4_train(s):
    xc, xs, xt, xct, xst, xtt = G.cast_nvfp4_pair(s["x"], s["hadamard"], None, None)
    wc, ws, wct, wst, wt = G.cast_nvfp4_square(s["w"])
    y = G.nvfp4_linear(xc, xs, wc, ws, (xt * wt).float(), s["one"], None)
    gc, gs, gt, gct, gst, gtt = G.cast_nvfp4_pair(s["g"], s["hadamard"], s["seeds"][0], s["seeds"][1])
    dx = G.nvfp4_linear(gc, gs, wct, wst, (gt * wt).float(), s["one"], None)
    dw = G.nvfp4_linear(gct, gst, xct, xst, (gtt * xtt).float(), s["one"], None)
    return y, dx, dw


_KINDS = {"mx_linear": (_prepare_mx_linear, _run_mx_linear), "fp8_layer": (_prepare_fp8_layer, _run_layer),
          "nvfp4_layer": (_prepare_nvfp4_layer, _run_layer), "decode": (_prepare_decode, _run_decode),
          "kivi": (_prepare_kivi, _run_kivi), "gptq": (_prepare_gptq, _run_gptq),
          "fp8_train": (_prepare_fp8_train, _run_fp8_train), "nvfp4_train": (_prepare_nvfp4_train, _run_nvfp4_train)}


def prepare(case, seed):
    with torch.no_grad():
        state = _KINDS[case["kind"]][0](case, seed)
    state["kind"] = case["kind"]
    return state


def run(state):
    with torch.no_grad():
        return _KINDS[state["kind"]][1](state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind, sh = case["kind"], SHAPE
    if kind == "mx_linear":
        m, n, k, block = case["tokens"], case["n"], case["k"], MX_FORMATS[case["format"]][1]
        return {"bytes": 2 * (m * k + n * k + n * k // block + m * n), "flops": 2.0 * m * n * k}
    params = sum(n * k for n, k in W.linear_shapes(sh).values())
    if kind in ("fp8_layer", "nvfp4_layer"):
        t, per = case["tokens"], 1.0 if kind == "fp8_layer" else 0.5625
        return {"bytes": per * params + 4 * t * sh.hidden,
                "flops": 2.0 * t * params + 2.0 * t * t * sh.heads * sh.head_dim}
    if kind == "decode":
        b, c, r = case["batch"], case["cached"], case["recent"]
        kv = b * sh.kv_heads * sh.head_dim
        cache = 2 * kv * (c // 4 + 4 * c // 64) + 2 * kv * r * 2
        return {"bytes": params * (0.5 + 2 / 64) + cache + 4 * b * sh.hidden,
                "flops": 2.0 * b * params + 4.0 * b * (c + r) * sh.heads * sh.head_dim}
    if kind == "kivi":
        values = 2 * case["batch"] * sh.kv_heads * case["positions"] * sh.head_dim
        return {"bytes": values * (2 + 2 + 0.25 + 4 / 64), "flops": 0.0}
    if kind == "gptq":
        n, k, t = case["n"], case["k"], case["tokens"]
        return {"bytes": 2 * t * k + 4 * k * k + 6 * n * k, "flops": float(t) * k * k + float(k) ** 3 + float(n) * k * k}
    m, n, k = case["tokens"], case["n"], case["k"]
    size = 2 * (m * k + n * k + m * n) * 2
    if kind == "fp8_train":
        size += 2 * m * k * 2      # the norm's input and the residual gradient
    return {"bytes": size, "flops": 6.0 * m * n * k}


def tolerance(case):
    return _TOLERANCE[case["kind"]]


# About four times what was measured between the path and another correct order of its sums.  One GEMM agrees with
# float64 operands' product to a handful of bfloat16 ties; a layer's later casts move whole codes on such a tie, more so
# the fewer bits they keep (fused against separate attention: FP8 0.4 %, NVFP4 1.6 %, MXNF4 decode 1.7 %); the GPTQ
# solve moved 1.1 % with a float64 Cholesky factor; the norm's weight gradient 0.02 %.
_TOLERANCE = {
    "mx_linear": {"rel": 1e-3, "max": 2e-2},
    "fp8_layer": {"rel": 1.5e-2, "max": 0.5},
    "nvfp4_layer": {"rel": 3e-2, "max": 0.95},
    "decode": {"rel": 3e-2, "max": 0.9},
    "kivi": "exact",
    "gptq": {"rel": 3e-2, "max": 0.95},
    "fp8_train": {"rel": 1e-3, "max": 8e-2},
    "nvfp4_train": {"rel": 1e-3, "max": 2e-2},
}
