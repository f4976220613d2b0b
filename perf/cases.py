"""The work this framework is used for, as measurable cases.

A case is a dict of plain values.  Kinds:
    step      one decode token (or a small batch of sequences) through the matrices of a transformer stack, one
              grouped launch: GroupedGemv
    layer     one packed Linear applied to `rows` activation rows: a single decode call, a speculative or small-batch
              call, a prompt of some thousand tokens
    mlp       a quantised stack of Linear layers evaluated as a model, fp32 activations, ungrouped codebooks
    conv      a quantised Conv2d of an image network, fp32 activations
    pack      quantisation of a dense fp32 matrix that is already on the GPU
    dequant   the dense fp32 matrix of a packed one (inspection, export, calibration code that asks for W_q)
"""
from __future__ import annotations

import math

import torch

import if_i_could_turn_back_time_b200 as jq

DEVICE = "cuda"
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
MOST_STEP_BYTES = 3.3e9      # of packed weights in a drawn step; the listed ones hold up to 3.45e9
MOST_FLOPS = 1.85e11         # of a drawn layer, mlp or conv; the largest listed layer has 1.85e11


def listed():
    return [
        # classifier of the pruning experiments: 784-300-100-10, one evaluation batch of 64 images
        {"name": "mlp_784_300_100_10", "kind": "mlp", "in": 784, "h1": 300, "h2": 100, "out": 10, "bias": False, "rows": 64},
        # one attention projection called by itself for one token: latency of a single call
        {"name": "layer_gf4_1", "kind": "layer", "fmt": "gf4", "g": 128, "had": 128, "N": 4096, "K": 4096, "rows": 1,
         "x": "bf16", "bias": False},
        # a down projection of the 7B shape for a ragged handful of sequences, with bias, fp16
        {"name": "layer_e2m1_23", "kind": "layer", "fmt": "e2m1", "g": 32, "had": 0, "N": 4096, "K": 11008, "rows": 23,
         "x": "fp16", "bias": True},
        # a decode token of the whole 7B-shaped stack, one sequence: the headline benchmark
        {"name": "step7b_gf4_1", "kind": "step", "fmt": "gf4", "g": 128, "had": 128, "layers": 32, "hidden": 4096, "kv": 4096,
         "ffn": 11008, "rows": 1},
        # the same stack serving eight sequences at once
        {"name": "step7b_gf4_8", "kind": "step", "fmt": "gf4", "g": 128, "had": 128, "layers": 32, "hidden": 4096, "kv": 4096,
         "ffn": 11008, "rows": 8},
        # the same stack in the E2M1 format, one sequence
        {"name": "step7b_e2m1_1", "kind": "step", "fmt": "e2m1", "g": 32, "had": 0, "layers": 32, "hidden": 4096, "kv": 4096,
         "ffn": 11008, "rows": 1},
        # seven of the 80 layers of the 70B-shaped stack (a pipeline stage), sixteen sequences
        {"name": "step70b_e2m1_16", "kind": "step", "fmt": "e2m1", "g": 32, "had": 0, "layers": 7, "hidden": 8192, "kv": 1024,
         "ffn": 28672, "rows": 16},
        # a prompt of 2048 tokens through a gate / up projection of the 7B shape
        {"name": "prefill_gf4_2048", "kind": "layer", "fmt": "gf4", "g": 128, "had": 128, "N": 11008, "K": 4096, "rows": 2048,
         "x": "bf16", "bias": False},
        # a ragged prompt through an attention projection of the 70B shape
        {"name": "prefill_e2m1_777", "kind": "layer", "fmt": "e2m1", "g": 32, "had": 0, "N": 8192, "K": 8192, "rows": 777,
         "x": "bf16", "bias": False},
        # a 3x3 convolution of an image network on a batch of feature maps
        {"name": "conv_64_128_3x3", "kind": "conv", "cin": 64, "cout": 128, "k": 3, "stride": 1, "pad": 1, "hw": 32, "batch": 16},
        # quantising an attention projection: rotation, group scales, per-row Jenks codebooks, codes
        {"name": "pack_gf4_4096", "kind": "pack", "fmt": "gf4", "g": 128, "had": 128, "N": 4096, "K": 4096},
        # the dense matrix of a packed gate / up projection
        {"name": "dequant_gf4_11008", "kind": "dequant", "fmt": "gf4", "g": 128, "had": 128, "N": 11008, "K": 4096},
    ]


# ---- drawn cases ---------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _format(rng):
    """A format as it is used in earnest: the default groups most of the time."""
    if rng.random() < 0.5:
        return "gf4", rng.choice([128, 128, 128, 128, 256, 64, 0]), rng.choice([0, 128])
    return "e2m1", rng.choice([32, 32, 32, 32, 64, 128]), rng.choice([0, 0, 128])


def _draw_step(rng):
    fmt, g, had = rng.choice([("gf4", 128, 128), ("gf4", 128, 0), ("e2m1", 32, 0), ("e2m1", 32, 128)])
    hidden = 256 * _log_int(rng, 4, 32)
    ffn = 256 * int(hidden * rng.uniform(2.5, 3.6) / 256)
    kv = hidden // rng.choice([1, 1, 4, 8])
    per_layer = (2 * hidden + 2 * kv) * hidden + 3 * hidden * ffn
    most = max(1, int(MOST_STEP_BYTES / (0.57 * per_layer)))
    return {"kind": "step", "fmt": fmt, "g": g, "had": had, "layers": _log_int(rng, 1, min(80, most)), "hidden": hidden,
            "kv": kv, "ffn": ffn, "rows": _log_int(rng, 1, 32)}


def _draw_layer(rng):
    fmt, g, had = _format(rng)
    N = _log_int(rng, 256, 28672)
    if rng.random() < 0.5:
        N = (N + 127) // 128 * 128      # half of them multiples of a tile, half ragged (a vocabulary, a pruned layer)
    unit = 256 if (g == 256 or rng.random() < 0.7) else 128
    K = unit * max(1, _log_int(rng, 512, 16384) // unit)
    most = max(1, min(4096, int(MOST_FLOPS / (2.0 * N * K))))
    return {"kind": "layer", "fmt": fmt, "g": g, "had": had, "N": N, "K": K, "rows": _log_int(rng, 1, most),
            "x": rng.choice(["bf16", "bf16", "fp16", "fp32"]), "bias": rng.random() < 0.4}


def _draw_mlp(rng):
    return {"kind": "mlp", "in": _log_int(rng, 64, 4096), "h1": _log_int(rng, 32, 2048), "h2": _log_int(rng, 32, 2048),
            "out": _log_int(rng, 10, 1000), "bias": rng.random() < 0.7, "rows": _log_int(rng, 1, 512)}


def _draw_conv(rng):
    k = rng.choice([1, 3, 3, 5])
    cin, cout = rng.choice([3, 16, 32, 48, 64, 96, 128, 256]), 8 * _log_int(rng, 1, 32)
    hw, stride = _log_int(rng, 7, 56), rng.choice([1, 1, 2])
    positions = (hw // stride) ** 2
    most = max(1, int(16 * 1024 * 576 / (positions * cin * k * k)))
    return {"kind": "conv", "cin": cin, "cout": cout, "k": k, "stride": stride, "pad": k // 2, "hw": hw,
            "batch": _log_int(rng, 1, min(64, most))}


def _draw_matrix(rng, kind):
    fmt, g, had = _format(rng)
    K = 256 * max(1, _log_int(rng, 512, 11008) // 256)
    N = _log_int(rng, 64, max(64, min(28672, int((4096 * 4096 if kind == "pack" else 11008 * 4096) / K))))
    return {"kind": kind, "fmt": fmt, "g": g, "had": had, "N": N, "K": K}


def draw(rng):
    r = rng.random()
    if r < 0.30:
        return _draw_step(rng)
    if r < 0.70:
        return _draw_layer(rng)
    if r < 0.78:
        return _draw_mlp(rng)
    if r < 0.86:
        return _draw_conv(rng)
    return _draw_matrix(rng, "pack" if r < 0.94 else "dequant")


# ---- states --------------------------------------------------------------------------------------------------------
def _weight(gen, N, K):
    """Dense weight of a trained layer as quantisers meet it: normal with a few outliers."""
    W = torch.randn(N, K, generator=gen, device=DEVICE) * 0.02
    W[torch.rand(N, K, generator=gen, device=DEVICE) < 1e-3] *= 8
    return W


def _module_weights(module, gen):
    with torch.no_grad():
        for m in module.modules():
            if isinstance(m, (torch.nn.Linear, torch.nn.Conv2d)):
                fan_in = m.weight[0].numel()
                m.weight.copy_(torch.randn(m.weight.shape, generator=gen, device=DEVICE) * fan_in ** -0.5)
                if m.bias is not None:
                    m.bias.copy_(torch.randn(m.bias.shape, generator=gen, device=DEVICE) * 0.1)


def _quantised(module):
    q = jq.quantize_module(module, 4, fmt="gf4", group_size=0)
    for m in q.modules():
        if hasattr(m, "commit"):
            m.commit()
    return q


def _stack_shapes(c):
    h, f, kv = c["hidden"], c["ffn"], c["kv"]
    return [(h, h), (kv, h), (kv, h), (h, h), (f, h), (f, h), (h, f)]      # q, k, v, o, gate, up, down


def prepare(case, seed):
    gen = torch.Generator(DEVICE).manual_seed(seed)
    kind = case["kind"]
    if kind == "step":
        spec = jq.QuantSpec(case["fmt"], case["g"], case["had"])
        proto = {}
        for shape in _stack_shapes(case):       # one matrix per distinct shape is quantised, every use has its own copy
            if shape not in proto:
                proto[shape] = jq.pack_weight(_weight(gen, *shape), spec)
        copy = lambda t: None if t is None else t.clone()
        weights = [jq.PackedWeight(p.spec, p.N, p.K, copy(p.qweight), copy(p.scales), copy(p.codebook))
                   for _ in range(case["layers"]) for p in (proto[s] for s in _stack_shapes(case))]
        grp = jq.ops.GroupedGemv(weights, case["rows"], torch.bfloat16)
        for x in grp.xs:
            x.copy_(torch.randn(x.shape, generator=gen, device=DEVICE))
        return {"kind": kind, "grp": grp}
    if kind == "layer":
        spec = jq.QuantSpec(case["fmt"], case["g"], case["had"])
        pw = jq.pack_weight(_weight(gen, case["N"], case["K"]), spec)
        x = torch.randn(case["rows"], case["K"], generator=gen, device=DEVICE).to(DTYPES[case["x"]])
        bias = torch.randn(case["N"], generator=gen, device=DEVICE) if case["bias"] else None
        return {"kind": kind, "x": x, "pw": pw, "bias": bias}
    if kind == "mlp":
        nn, b = torch.nn, case["bias"]
        model = nn.Sequential(nn.Flatten(), nn.Linear(case["in"], case["h1"], bias=b), nn.ReLU(),
                              nn.Linear(case["h1"], case["h2"], bias=b), nn.ReLU(),
                              nn.Linear(case["h2"], case["out"], bias=b)).to(DEVICE)
        _module_weights(model, gen)
        x = torch.rand(case["rows"], case["in"], generator=gen, device=DEVICE)      # pixel values
        return {"kind": kind, "model": _quantised(model), "x": x}
    if kind == "conv":
        conv = torch.nn.Conv2d(case["cin"], case["cout"], case["k"], stride=case["stride"], padding=case["pad"]).to(DEVICE)
        _module_weights(conv, gen)
        x = torch.randn(case["batch"], case["cin"], case["hw"], case["hw"], generator=gen, device=DEVICE).relu_()
        return {"kind": kind, "model": _quantised(conv), "x": x}
    spec = jq.QuantSpec(case["fmt"], case["g"], case["had"])
    W = _weight(gen, case["N"], case["K"])
    if kind == "pack":
        return {"kind": kind, "W": W, "spec": spec}
    return {"kind": kind, "pw": jq.pack_weight(W, spec)}


def run(state):
    kind = state["kind"]
    if kind == "step":
        grp = state["grp"]
        grp.run()
        return grp.y_arena.view(torch.bfloat16)         # all outputs of the step, one arena
    if kind == "layer":
        return jq.ops.linear(state["x"], state["pw"], state["bias"])
    if kind in ("mlp", "conv"):
        with torch.no_grad():
            return state["model"](state["x"])
    if kind == "pack":
        pw = jq.pack_weight(state["W"], state["spec"])
        return {"qweight": pw.qweight, "scales": pw.scales, "codebook": pw.codebook}
    return jq.ops.dequantize(state["pw"])


# ---- what a pass cannot do without ---------------------------------------------------------------------------------
def _linear_work(spec, N, K, rows, xb, yb, bias):
    return {"bytes": jq.algorithmic_bytes(spec, N, K, rows, xb, yb, bias), "flops": 2.0 * N * K * rows}


def _sum(works):
    return {"bytes": sum(w["bytes"] for w in works), "flops": sum(w["flops"] for w in works)}


def work(case):
    kind = case["kind"]
    if kind == "step":
        spec = jq.QuantSpec(case["fmt"], case["g"], case["had"])
        return _sum([_linear_work(spec, n, k, case["rows"], 2, 2, False) for n, k in _stack_shapes(case)] * case["layers"])
    if kind == "layer":
        spec = jq.QuantSpec(case["fmt"], case["g"], case["had"])
        size = DTYPES[case["x"]].itemsize
        return _linear_work(spec, case["N"], case["K"], case["rows"], size, size, case["bias"])
    if kind == "mlp":
        spec = jq.QuantSpec("gf4", 0, 0)
        dims = [case["in"], case["h1"], case["h2"], case["out"]]
        w = _sum([_linear_work(spec, n, k, case["rows"], 0, 0, case["bias"]) for k, n in zip(dims, dims[1:])])
        return {"bytes": w["bytes"] + 4.0 * case["rows"] * (case["in"] + case["out"]), "flops": w["flops"]}
    if kind == "conv":
        kc, out = case["cin"] * case["k"] ** 2, (case["hw"] + 2 * case["pad"] - case["k"]) // case["stride"] + 1
        w = _linear_work(jq.QuantSpec("gf4", 0, 0), case["cout"], kc, case["batch"] * out * out, 0, 4, True)
        return {"bytes": w["bytes"] + 4.0 * case["batch"] * case["cin"] * case["hw"] ** 2, "flops": w["flops"]}
    spec = jq.QuantSpec(case["fmt"], case["g"], case["had"])
    packed = jq.algorithmic_bytes(spec, case["N"], case["K"], 0, 0, 0)
    return {"bytes": packed + 4.0 * case["N"] * case["K"], "flops": 0.0}


def tolerance(case):
    """Quantised tensors and dequantised weights are defined bit for bit.  Products round the activation to fp16 (and,
    for larger E2M1 batches, the scaled weight) and the result to its own type.  Against the same product in 64 bits
    that comes to 1.7e-3 for bf16 results, 3.4e-4 for fp16, 2.7e-4 for fp32 and 4.3e-4 after three fp32 layers; the
    limits are four times that."""
    kind = case["kind"]
    if kind in ("pack", "dequant"):
        return "exact"
    if kind == "mlp":
        return {"rel": 1.7e-3}
    out = "bf16" if kind == "step" else case.get("x", "fp32")
    return {"rel": {"bf16": 7e-3, "fp16": 1.4e-3, "fp32": 1.1e-3}[out]}


# ---- the same results in 64 bits, plain torch ----------------------------------------------------------------------
E2M1_VALUES = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0)


def _dense64(pw):
    """The weight matrix that the packed tensors stand for: value or codebook entry, times the scale of its group."""
    byte = pw.qweight.long()
    code = torch.stack([byte & 15, byte >> 4], dim=2).reshape(pw.N, -1)[:, :pw.K]
    if pw.spec.fmt == "e2m1":
        w = torch.tensor(E2M1_VALUES, dtype=torch.float64, device=DEVICE)[code]
    else:
        w = torch.gather(pw.codebook.double(), 1, code)
    if pw.scales is not None:
        w.view(pw.N, -1, pw.spec.group_size).mul_(pw.scales.double()[:, :, None])
    return w


def _hadamard64(n):
    h = torch.ones(1, 1, dtype=torch.float64, device=DEVICE)
    while h.shape[0] < n:
        h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
    return h / n ** 0.5


def _linear64(x, pw, bias=None):
    x = x.double()
    if pw.spec.had_block:
        b = pw.spec.had_block
        x = (x.reshape(-1, pw.K // b, b) @ _hadamard64(b)).reshape(-1, pw.K)
    y = x @ _dense64(pw).t()
    return y if bias is None else y + bias.double()


def exact(case, seed):
    """Quantising has no value besides the one that the format defines; everything else is a product in 64 bits."""
    kind = case["kind"]
    if kind == "pack":
        return None
    s = prepare(case, seed)
    if kind == "dequant":
        return _dense64(s["pw"])
    if kind == "layer":
        return _linear64(s["x"], s["pw"], s["bias"])
    if kind == "step":
        grp = s["grp"]
        y = torch.zeros(grp.y_arena.numel() // 2, dtype=torch.float64, device=DEVICE)
        for x, w, o in zip(grp.xs, grp.weights, grp.y_offsets):
            y[o // 2:o // 2 + case["rows"] * w.N] = _linear64(x, w).reshape(-1)
        return y
    if kind == "conv":
        m, x = s["model"], s["x"]
        w = _dense64(m.packed).reshape(m.out_channels, m.in_channels, *m.kernel_size)
        return torch.nn.functional.conv2d(x.double(), w, m.bias.double(), m.stride, m.padding)
    x = s["x"].double()
    for m in s["model"]:
        if isinstance(m, torch.nn.Linear):
            x = _linear64(x, m.packed, m.bias)
        elif isinstance(m, torch.nn.ReLU):
            x = x.relu()
    return x
