"""What this package is measured on: the calls that a program on top of it makes, over the sizes it makes them with.

Four kinds of work, each through the public entry points in `ac4k_kernel_b200.ops`:

  linear     a linear layer: the bf16 activations are quantised and multiplied with a weight that was quantised when the
             model was loaded (`quantize` -> `linear`, or `-> linear_requant` where the next layer takes NVFP4)
  quantize   a tensor quantised by itself, to NVFP4, per-token FP8 or per-token INT8 (weights, caches, activations)
  attention  one attention layer on bf16 q, k, v (the quantisers and the attention kernel), in both precisions
  rope       the 3-D rotary embedding of q or k
"""
import math

import torch

from ac4k_kernel_b200 import ops

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_MAX_GEMM = 8192 * 28672 * 8192            # M * N * K of the largest linear layer
_MAX_ELEMENTS = 32768 * 8192               # of the largest tensor that is quantised by itself
_MAX_SCORES = 40 * 75600 * 75600           # B * H * Nq * Nkv of the largest attention layer
_MAX_ROPE = 75600 * 40 * 128


def _linear(name, m, n, k, layout="ac4k", bias=False, out="bf16"):
    return {"name": name, "kind": "linear", "m": m, "n": n, "k": k, "layout": layout, "bias": bias, "out": out}


def _quantize(name, rows, cols, precision, layout="ac4k"):
    return {"name": name, "kind": "quantize", "rows": rows, "cols": cols, "precision": precision, "layout": layout}


def _attention(name, b, h, nq, nkv, d, precision, layout="BNHD"):
    return {"name": name, "kind": "attention", "b": b, "h": h, "nq": nq, "nkv": nkv, "d": d, "precision": precision,
            "layout": layout}


def _rope(name, b, f, h, w, heads, d):
    return {"name": name, "kind": "rope", "b": b, "f": f, "h": h, "w": w, "heads": heads, "d": d}


def listed():
    return [
        # one token of one sequence through a projection: the smallest call, its launches and its weight stream
        _linear("decode_1", 1, 8192, 8192),
        # a decode batch that fills no tile, the scales in the tensor-memory layout, with a bias
        _linear("decode_50", 50, 8192, 8192, layout="128x4", bias=True),
        # a prompt of odd length: ragged row tiles, too few of them for the chip
        _linear("prefill_666", 666, 4096, 4096, bias=True),
        # the square GEMM that this library is quoted on, with the quantisation of its activations
        _linear("square_4096", 4096, 4096, 4096, layout="128x4"),
        # the up projection of an MLP in prefill: the largest GEMM
        _linear("mlp_8192", 8192, 28672, 8192),
        # a layer whose output the next layer takes in NVFP4
        _linear("requant_2048", 2048, 8192, 4096, layout="128x4", out="nvfp4"),
        # a whole activation or weight tensor to NVFP4, global scale included
        _quantize("quantize_nvfp4", 32768, 8192, "nvfp4"),
        # per-token FP8 of a mid-size activation tensor with an odd number of rows
        _quantize("quantize_fp8", 4099, 5120, "fp8e4m3"),
        # video self-attention at 21 x 45 x 80 positions, the default precision: the largest attention
        _attention("attention_int8_75600", 1, 40, 75600, 75600, 128, "int8+fp8e4m3"),
        # a long sequence in the NVFP4 precision
        _attention("attention_nvfp4_16384", 1, 16, 16384, 16384, 128, "nvfp4"),
        # many short sequences with an odd head dimension
        _attention("attention_int8_100", 11, 12, 100, 100, 65, "int8+fp8e4m3"),
        # the rotary embedding of the video's q or k
        _rope("rope_75600", 1, 21, 45, 80, 40, 128),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _to(x, multiple):
    return max(multiple, x // multiple * multiple)


def draw(rng):
    kind = rng.choices(["linear", "quantize", "attention", "rope"], [5, 2, 4, 1])[0]
    if kind == "linear":
        # rows: any number of tokens; features: multiples of 64 as layers have them, now and then only of 8
        m = _log(rng, 1, 8192)
        n, k = (_to(_log(rng, 512, 28672), rng.choice([64, 64, 64, 8])) for _ in range(2))
        k = min(k, 16384)
        while m * n * k > _MAX_GEMM:
            m //= 2
        out = rng.choices(["bf16", "fp16", "fp32", "nvfp4"], [12, 1, 1, 2])[0]
        if out == "nvfp4":
            n = _to(n, 64)
        return {"kind": kind, "m": m, "n": n, "k": k, "layout": rng.choice(["ac4k", "128x4"]), "bias": rng.random() < 0.4,
                "out": out}
    if kind == "quantize":
        cols = _to(_log(rng, 512, 16384), rng.choice([64, 64, 16]))
        rows = min(_log(rng, 1, 32768), _MAX_ELEMENTS // cols)
        return {"kind": kind, "rows": rows, "cols": cols, "precision": rng.choice(["nvfp4", "fp8e4m3", "int8"]),
                "layout": rng.choice(["ac4k", "128x4"])}
    if kind == "attention":
        h, d = _log(rng, 1, 40), rng.choice([64, 80, 96, 100, 128, 128, 128, 128])
        nq = _log(rng, 64, 75600)
        nkv = nq if rng.random() < 0.75 else _log(rng, 64, 8192)       # self attention, or against a text or image context
        b = rng.choice([1, 1, 2, 4, 11]) if nq <= 4096 else 1
        while b * h * nq * nkv > _MAX_SCORES or b * h * max(nq, nkv) * d > _MAX_ROPE:
            nq, nkv = nq // 2, nkv // 2
        return {"kind": kind, "b": b, "h": h, "nq": nq, "nkv": nkv, "d": d, "precision": rng.choice(["int8+fp8e4m3", "nvfp4"]),
                "layout": rng.choice(["BNHD", "BNHD", "BHND"])}
    f, hh, w = _log(rng, 1, 21), _log(rng, 4, 45), _log(rng, 5, 80)
    return {"kind": kind, "b": rng.choice([1, 1, 2]) if f * hh * w <= 32768 else 1, "f": f, "h": hh, "w": w,
            "heads": _log(rng, 5, 40), "d": rng.choice([64, 96, 128, 128])}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(shape, g):
    """N(0, 1) with half a percent of outliers thirty times as large, as hidden states have them."""
    x = torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16)
    return torch.where(torch.rand(shape, generator=g, device="cuda", dtype=torch.float16) < 0.005, x * 30, x)


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        weight = torch.randn((n, k), generator=g, device="cuda", dtype=torch.bfloat16) * 0.02
        state = {"case": case, "x": _activations((m, k), g), "weight": ops.quantize(weight, 0, 1, sf_layout=case["layout"]),
                 "bias": torch.randn((n,), generator=g, device="cuda", dtype=torch.bfloat16) if case["bias"] else None}
        if case["out"] == "nvfp4":
            # a calibrated scale: the standard deviation of the outputs is known, six of it are the largest value
            sigma = 0.02 * math.sqrt(k * (1 + 0.005 * 900))
            state["out_scale"] = torch.full((), 6 * sigma / (6.0 * 448.0), dtype=torch.float32, device="cuda")
        return state
    if kind == "quantize":
        return {"case": case, "x": _activations((case["rows"], case["cols"]), g)}
    if kind == "attention":
        b, h, d = case["b"], case["h"], case["d"]

        def tensor(n):
            shape = (b, n, h, d) if case["layout"] == "BNHD" else (b, h, n, d)
            return torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16)

        # keys share an offset per channel, which the INT8 path takes off before it quantises them
        k = tensor(case["nkv"])
        k += torch.randn((h, d) if case["layout"] == "BNHD" else (h, 1, d), generator=g, device="cuda", dtype=torch.bfloat16)
        return {"case": case, "q": tensor(case["nq"]), "k": k, "v": tensor(case["nkv"])}
    b, f, h, w, d = case["b"], case["f"], case["h"], case["w"], case["d"]
    x = torch.randn((b, f * h * w, case["heads"], d), generator=g, device="cuda", dtype=torch.bfloat16)

    def angles(pairs):
        position = torch.arange(1024, dtype=torch.float64, device="cuda")
        return torch.outer(position, 10000.0 ** (-torch.arange(pairs, dtype=torch.float64, device="cuda") / pairs))

    c = d // 2
    parts = [c - 2 * (c // 3), c // 3, c // 3]                 # frame, height and width
    angle = torch.cat([angles(p) for p in parts], dim=1)
    return {"case": case, "x": x, "grid": torch.tensor([[f, h, w]] * b, dtype=torch.int32, device="cuda"),
            "freqs": torch.polar(torch.ones_like(angle), angle)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        w, w_sf, w_scale = state["weight"]
        x, x_sf, x_scale = ops.quantize(state["x"], 0, 1, sf_layout=case["layout"])
        if case["out"] == "nvfp4":
            return ops.linear_requant(x, x_sf, x_scale, w, w_sf, w_scale, state["out_scale"], bias=state["bias"],
                                      sf_layout=case["layout"])
        if case["out"] == "bf16":
            return ops.linear(x, x_sf, x_scale, w, w_sf, w_scale, bias=state["bias"])
        out = torch.empty((case["m"], case["n"]), dtype=_DTYPES[case["out"]], device="cuda")
        return ops.linear(x, x_sf, x_scale, w, w_sf, w_scale, bias=state["bias"], out=out)
    if kind == "quantize":
        if case["precision"] == "nvfp4":
            return ops.quantize(state["x"], 0, 1, sf_layout=case["layout"])
        return ops.quantize(state["x"], 0, 1, precision=case["precision"])
    if kind == "attention":
        return ops.attention(state["q"], state["k"], state["v"], layout=case["layout"], precision=case["precision"])
    return ops.rope3d(state["x"], state["grid"], state["freqs"])


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        out = {"bf16": 2, "fp16": 2, "fp32": 4, "nvfp4": 9 / 16}[case["out"]]
        return {"bytes": 2 * m * k + 9 / 16 * n * k + out * m * n + (2 * n if case["bias"] else 0), "flops": 2 * m * n * k}
    if kind == "quantize":
        out = {"nvfp4": 9 / 16, "fp8e4m3": 1, "int8": 1}[case["precision"]]
        scales = 0 if case["precision"] == "nvfp4" else 4 * case["rows"]
        return {"bytes": (2 + out) * case["rows"] * case["cols"] + scales, "flops": 0}
    if kind == "attention":
        b, h, nq, nkv, d = (case[key] for key in ("b", "h", "nq", "nkv", "d"))
        return {"bytes": 4 * b * h * d * (nq + nkv), "flops": 4 * b * h * nq * nkv * d}
    elements = case["b"] * case["f"] * case["h"] * case["w"] * case["heads"] * case["d"]
    return {"bytes": 4 * elements, "flops": 3 * elements}


def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        # against sums in 64 bits: 3e-8 in fp32, 6e-6 where a sum's last bits move a rounding to 16 bits; no code of a
        # re-quantised output moved, a single block scale that does is 6e-5 of a small output
        if case["out"] == "nvfp4":
            return {"rel": 2e-4, "differ": 1e-4}
        return {"rel": 1e-6 if case["out"] == "fp32" else 1e-4}
    if kind == "attention":
        # against the sums in another order and exp2 instead of its approximation: 1e-3 where roundings of P and of the
        # result move; 2e-3 in the INT8 path where the mean that is taken off the keys moves by a bit of bf16
        return {"rel": 4e-3 if case["precision"] == "nvfp4" else 8e-3}
    return "exact"                                             # quantisers and the rotary embedding: bit for bit


def _nvfp4(x):
    """x [rows, columns] to NVFP4 and back, in 64 bits: one scale for the tensor, an e4m3 scale per block of 16, e2m1 values."""
    rows, cols = x.shape
    x = torch.nn.functional.pad(x.float(), (0, -cols % 16)).reshape(rows, -1, 16)
    amax = x.abs().amax(dim=2, keepdim=True)
    scale = amax.max() / 2688.0
    block = ((1.0 / scale) * (amax * (1.0 / 6.0))).clamp(max=448.0).to(torch.float8_e4m3fn).float()
    a = torch.where(block > 0, x * ((1.0 / scale) * (1.0 / block)), torch.zeros_like(x))
    code = torch.zeros(a.shape, dtype=torch.int64, device=a.device)
    for at, up in ((0.25, False), (0.75, True), (1.25, False), (1.75, True), (2.5, False), (3.5, True), (5.0, False)):
        code += (a.abs() >= at) if up else (a.abs() > at)         # a tie goes to the value of even mantissa
    value = torch.tensor([0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0], dtype=torch.float64, device=a.device)[code]
    return (value * a.sign() * block.double() * scale.double()).reshape(rows, -1)[:, :cols], scale


def exact(case, seed):
    """What `run` gives for these inputs, in 64 bits; None in the place of packed bytes and their block scales."""
    g = _generator(seed)
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        if case["out"] == "nvfp4":
            return None, None, prepare(case, seed)["out_scale"].double()
        weight = torch.randn((n, k), generator=g, device="cuda", dtype=torch.bfloat16) * 0.02
        x = _activations((m, k), g)
        y = _nvfp4(x)[0] @ _nvfp4(weight)[0].T
        if case["bias"]:
            y += torch.randn((n,), generator=g, device="cuda", dtype=torch.bfloat16)
        return y
    if kind == "quantize":
        x = _activations((case["rows"], case["cols"]), g)
        if case["precision"] == "nvfp4":
            return None, None, x.abs().max().double() / 2688.0
        scale = x.abs().amax(dim=1).double() / (448.0 if case["precision"] == "fp8e4m3" else 127.0)
        return None, torch.nn.functional.pad(scale, (0, -case["rows"] % 16))
    if kind == "attention":
        # four-bit probabilities are further than a tenth from the exact ones; the longest take too long in 64 bits
        if case["precision"] == "nvfp4" or case["b"] * case["h"] * case["nq"] * case["nkv"] > 2e10:
            return None
        state = prepare(case, seed)
        q, k, v = (state[name] if case["layout"] == "BHND" else state[name].transpose(1, 2) for name in ("q", "k", "v"))
        out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
        step = max(1, 2 ** 28 // case["nkv"])
        for b in range(case["b"]):
            for h in range(case["h"]):
                kt, vt = k[b, h].double().T, v[b, h].double()
                for i in range(0, case["nq"], step):
                    out[b, h, i:i + step] = torch.softmax(q[b, h, i:i + step].double() @ kt / math.sqrt(case["d"]), dim=1) @ vt
        return out if case["layout"] == "BHND" else out.transpose(1, 2)
    state = prepare(case, seed)
    x, freqs = state["x"], state["freqs"]
    f, h, w = case["f"], case["h"], case["w"]
    c = case["d"] // 2
    parts = freqs.split([c - 2 * (c // 3), c // 3, c // 3], dim=1)
    turn = torch.cat([parts[0][:f].view(f, 1, 1, -1).expand(f, h, w, -1), parts[1][:h].view(1, h, 1, -1).expand(f, h, w, -1),
                      parts[2][:w].view(1, 1, w, -1).expand(f, h, w, -1)], dim=-1).reshape(f * h * w, 1, c)
    out = torch.empty(x.shape, dtype=torch.float64, device="cuda")
    for b in range(case["b"]):
        out[b] = torch.view_as_real(torch.view_as_complex(x[b].double().reshape(f * h * w, case["heads"], c, 2)) * turn).flatten(2)
    return out
