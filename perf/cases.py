"""Performance cases: the work this library is used for, through its public Python entry points.

Three kinds of program stand behind them.

* Serving one quantized layer: a program keeps `QuantizedLinear` / `QuantizedLinear4Bit` modules (packed codes, scales,
  bias, scratch) and calls them eagerly, with 1 .. 16 rows per call while tokens are decoded, a few dozen rows when
  requests are batched, and 64 .. 8192 rows for prompts; weights stored [in, out] (the modules' default) or [out, in],
  INT8 per row / per tensor or INT4 in groups of 32, 64 or 128, with and without a bias.  `linear_w8a8` is the same
  with INT8 activations, `quantized_matmul_backward_x` the gradient into the activations of a frozen layer.
* Packing: quantizing weights when a checkpoint is converted, and dequantizing them when one is exported.
* Generation: a whole NanoLLaMA-INT4 greedy generation, prompt and decode steps.

Sizes are those of the benchmark configurations (1024 x 1024, 4096 x 4096, 11008 x 4096, 28672 x 8192, the decoder of
dim 2048 / hidden 5632 / vocabulary 32000) and generic ones around them; `draw` spreads over the ranges in between.
"""
from __future__ import annotations

import importlib
import math

import torch

sgq = importlib.import_module("soverign-grad_b200")             # the directory name is not a Python identifier
nanollama = importlib.import_module("soverign-grad_b200.nanollama")

MAX_WEIGHT = 28672 * 8192           # elements of the largest weight
MAX_FLOPS = 2 * 8192 * MAX_WEIGHT   # of the largest single layer call


def _layer(name, m, k, n, bits, layout, group=32, scheme="row", bias=False, kind="forward"):
    return {"name": name, "kind": kind, "m": m, "k": k, "n": n, "bits": bits, "layout": layout, "group": group if bits == 4 else 0,
            "scheme": scheme if bits == 8 else "", "bias": bias}


def listed():
    return [
        # one sequence's token through the smallest module: nothing but call, launch and latency
        _layer("token_module_1024_m1", 1, 1024, 1024, 8, "kn", bias=True),
        # one sequence's token through a feed-forward up projection stored [out, in]: the benchmark's decode workload
        _layer("token_int4_11008x4096_m1", 1, 4096, 11008, 4, "nk"),
        # a small batch's tokens through the same projection as the modules store it by default ([in, out])
        _layer("token_module_int4_m4", 4, 4096, 11008, 4, "kn", bias=True),
        # a full decode batch through the largest layer, INT8: 235 MB of weights per call
        _layer("token_int8_28672x8192_m16", 16, 8192, 28672, 8, "nk", scheme="tensor"),
        # requests batched beyond a decode batch, below a prompt
        _layer("batch_int4_4096_m40", 40, 4096, 4096, 4, "nk"),
        # a ragged prompt through a module in its default layout
        _layer("prompt_module_int8_m1000", 1000, 4096, 11008, 8, "kn", bias=True),
        # long prompts packed together through the largest layer
        _layer("prompt_int4_28672x8192_m8192", 8192, 8192, 28672, 4, "nk"),
        # a prompt with INT8 activations
        _layer("prompt_w8a8_11008x4096", 2048, 4096, 11008, 8, "nk", kind="w8a8"),
        # gradient through a frozen module (adapter training in front of a quantized layer)
        _layer("grad_module_int4_m2048", 2048, 4096, 11008, 4, "kn", kind="backward"),
        # checkpoint conversion: one feed-forward weight to INT4 ...
        {"name": "pack_int4_11008x4096", "kind": "pack", "rows": 11008, "cols": 4096, "bits": 4, "group": 32, "scheme": ""},
        # ... and an attention weight back from INT8
        {"name": "unpack_int8_4096x4096", "kind": "unpack", "rows": 4096, "cols": 4096, "bits": 8, "group": 0, "scheme": "tensor"},
        # the decoder of the benchmark: eight prompts of 512 tokens, 128 greedy tokens each
        {"name": "generate_b8_p512_n128", "kind": "generate", "batch": 8, "prompt": 512, "new": 128, "layers": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(v, of, lo):
    return max(lo, v // of * of)


def draw(rng):
    """One more case of the same ranges.  Inner sizes are multiples of 64, output sizes of the [in, out] layout multiples
    of the group (what the modules are built with); everything else may be odd."""
    kind = rng.choices(["token", "batch", "prompt", "w8a8", "backward", "pack", "unpack", "generate"], [30, 10, 22, 8, 8, 10, 6, 6])[0]
    if kind == "generate":
        return {"kind": kind, "batch": rng.randint(1, 8), "prompt": _log_int(rng, 16, 512), "new": _log_int(rng, 8, 128),
                "layers": rng.randint(2, 16)}
    bits = rng.choice([4, 8])
    if kind in ("pack", "unpack"):
        cols = _log_int(rng, 1000, 8192)
        cols = cols if rng.random() < 0.3 else _multiple(cols, 128, 128)
        return {"kind": kind, "rows": min(_log_int(rng, 512, 28672), MAX_WEIGHT // cols), "cols": cols, "bits": bits,
                "group": rng.choice([32, 32, 64, 128]) if bits == 4 else 0, "scheme": rng.choice(["tensor", "row"]) if bits == 8 else ""}
    m = {"token": lambda: _log_int(rng, 1, 16), "batch": lambda: rng.randint(17, 63)}.get(kind, lambda: _log_int(rng, 64, 8192))()
    layout = rng.choice(["kn", "nk"])
    group = rng.choice([32, 32, 32, 64, 128])
    k = _multiple(_log_int(rng, 1024, 8192), rng.choice([64, 256, 256, 256]), 1024)
    n = min(_log_int(rng, 1000, 28672), MAX_WEIGHT // k)
    if kind == "w8a8":
        bits, layout = 8, "nk"
    elif layout == "kn" or kind == "backward":
        n = _multiple(n, max(64, group), 1024)
    elif rng.random() < 0.7:
        n = _multiple(n, 16, 16)
    c = _layer("", m, k, n, bits, layout, group, rng.choice(["tensor", "row"]), rng.random() < 0.5,
               kind if kind in ("w8a8", "backward") else "forward")
    del c["name"]
    if c["kind"] == "backward":
        c["bias"] = False
    return c


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(rows, width, gen):
    """N(0, 1) rows in which a few channels (one in 512, the same for every row) are twenty times larger, as those of a
    normalised decoder activation are."""
    x = torch.randn(rows, width, device="cuda", generator=gen)
    hot = torch.randint(0, width, (max(1, width // 512),), device="cuda", generator=gen)
    x[:, hot] *= 20.0
    return x


def _decoder_init(cfg, gen):
    """Random weights with the reference's Linear initialiser; the embedding is N(0, 1) and the output head a permutation
    of it, so that the model is as sure of its next token as a trained one is (tokens do not hang on rounding)."""
    made = {}

    def make(name, layer):
        out_f, in_f = nanollama.weight_shape(cfg, name)
        if name == "embed":
            made[name] = torch.randn(out_f, in_f, device="cuda", generator=gen)
            return made[name]
        std = math.sqrt(2.0 / (in_f + out_f))
        if name == "lm_head":
            return made.pop("embed")[torch.randperm(out_f, device="cuda", generator=gen)] * std
        return torch.randn(out_f, in_f, device="cuda", generator=gen) * std
    return make


def _scheme(case):
    return sgq.PER_TENSOR if case["scheme"] == "tensor" else sgq.PER_ROW


def _quantize(w, case):
    return sgq.quantize_int4(w, case["group"]) if case["bits"] == 4 else sgq.quantize_int8(w, _scheme(case))


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "generate":
        cfg = nanollama.NanoLlamaConfig(n_layers=case["layers"])
        model = nanollama.NanoLlamaInt4(cfg, "cuda", case["batch"], init=_decoder_init(cfg, gen))
        prompt = torch.randint(0, cfg.vocab, (case["batch"], case["prompt"]), device="cuda", generator=gen)
        return {"kind": kind, "model": model, "prompt": prompt, "new": case["new"]}
    if kind in ("pack", "unpack"):
        w = torch.randn(case["rows"], case["cols"], device="cuda", generator=gen) * 0.02
        w *= torch.where(torch.rand(w.shape, device="cuda", generator=gen) < 0.01, 20.0, 1.0)       # 1 % outliers
        if kind == "unpack":
            return {"kind": kind, "q": _quantize(w, case), "bits": case["bits"]}
        return {"kind": kind, "w": w, "case": dict(case)}
    m, k, n = case["m"], case["k"], case["n"]
    layout = sgq.LAYOUT_KN if case["layout"] == "kn" else sgq.LAYOUT_NK
    w = torch.randn((k, n) if case["layout"] == "kn" else (n, k), device="cuda", generator=gen) * 0.02
    bias = torch.randn(n, device="cuda", generator=gen) * 0.1 if case["bias"] else None
    if kind == "backward":
        return {"kind": kind, "q": _quantize(w, case), "layout": layout, "workspace": sgq.Workspace(torch.device("cuda")),
                "dy": torch.randn(m, n, device="cuda", generator=gen)}
    x = _activations(m, k, gen)
    if kind == "w8a8":
        return {"kind": kind, "q": _quantize(w, case), "bias": bias, "x": x}
    if case["bits"] == 4:
        layer = sgq.QuantizedLinear4Bit.from_float(w, bias, case["group"], layout)
    else:
        layer = sgq.QuantizedLinear.from_float(w, bias, _scheme(case), layout)
    return {"kind": kind, "layer": layer, "x": x}


def run(state):
    kind = state["kind"]
    if kind == "forward":
        return state["layer"](state["x"])
    if kind == "w8a8":
        return sgq.linear_w8a8(state["x"], state["q"], state["bias"])
    if kind == "backward":
        return sgq.quantized_matmul_backward_x(state["dy"], state["q"], layout=state["layout"], workspace=state["workspace"])
    if kind == "pack":
        q = _quantize(state["w"], state["case"])
        return q.qdata, q.scales
    if kind == "unpack":
        return sgq.dequantize_int4(state["q"]) if state["bits"] == 4 else sgq.dequantize_int8(state["q"])
    model = state["model"]
    tokens = model.generate(state["prompt"], state["new"])
    return {"tokens": tokens, "k_cache": model.k_cache, "v_cache": model.v_cache}


def _packed_bytes(rows, cols, bits, group, scheme):
    if bits == 4:
        return (rows * cols + 1) // 2 + 4 * -(-rows * cols // group)
    return rows * cols + 4 * (1 if scheme == "tensor" else rows)


def work(case):
    kind = case["kind"]
    if kind in ("pack", "unpack"):
        numel = case["rows"] * case["cols"]
        return {"bytes": 4 * numel + _packed_bytes(case["rows"], case["cols"], case["bits"], case["group"], case["scheme"]), "flops": 0}
    if kind == "generate":
        c = nanollama.NanoLlamaConfig(n_layers=case["layers"])
        b, p, steps = case["batch"], case["prompt"], case["new"] - 1
        layer = 4 * c.dim * c.dim + 3 * c.dim * c.hidden            # weights of one block
        head = c.vocab * c.dim
        weight_bytes = (c.n_layers * layer + head) * (0.5 + 4 / 32)
        cached = sum(p + i for i in range(steps))                   # positions read over all steps, per sequence
        kv_row = c.n_layers * 2 * c.dim * 4
        nbytes = (1 + steps) * weight_bytes + b * kv_row * (2 * p + cached + steps) + b * (p + steps) * c.dim * 4
        flops = 2 * b * ((p + steps) * c.n_layers * layer + (1 + steps) * head)
        flops += 4 * b * c.n_layers * c.dim * (p * (p + 1) // 2 + cached + steps)
        return {"bytes": nbytes, "flops": flops}
    m, k, n = case["m"], case["k"], case["n"]
    rows, cols = (k, n) if case["layout"] == "kn" else (n, k)
    nbytes = _packed_bytes(rows, cols, case["bits"], case["group"], case["scheme"]) + 4 * m * (k + n) + (4 * n if case["bias"] else 0)
    return {"bytes": nbytes, "flops": 2 * m * k * n}


def tolerance(case):
    kind = case["kind"]
    if kind in ("pack", "unpack"):
        return "exact"                                  # codes, bytes and scales are the reference's, bit for bit
    if kind == "generate":
        return {"rel": 1e-2, "differ": 0.005}           # bf16 products in the prompt pass
    if kind == "w8a8":
        return {"rel": 1e-6}                            # exact integer sums, then three fp32 roundings
    if case["m"] >= 64:
        return {"rel": 1e-2}                            # bf16 products
    if case["m"] >= 3 and case["layout"] == "nk":
        return {"rel": 1e-4}                            # activations held to 16 bits below the absmax of a group
    return {"rel": 1e-5}                                # fp32 sums
