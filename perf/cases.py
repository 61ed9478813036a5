"""Performance cases of the calibrate-and-quantize path, at the sizes its users run it at.

Five entry points, each as a user's program calls it:

``rtn``      ``oneshot`` with a ``QuantizationModifier`` (no calibration data) on sibling Linear modules, then
             ``compress_state_dict`` of each: what a data-free quantisation does per module.
``awq``      ``scaled_fake_quantize``: one grid point of the AWQ scale search on the layers behind one norm.
``hessian``  ``make_empty_hessian``, ``accumulate_hessian_lower`` per calibration batch, ``finalize_hessian``.
``gptq``     the same Hessian, then ``quantize_weight`` and ``compress_state_dict`` of one module.
``layer``    ``GPTQModifier`` over the calibration batches of one decoder layer, or of one layer's experts:
             hook calls per module and batch, then the end of the sequential epoch.

Weights are N(0, 0.02) in bfloat16 (``rtn`` adds 0.1 % N(0, 0.5) outliers, as checkpoints have them);
activations are normal with a scale of their own per channel.
"""
from __future__ import annotations

import math

import torch

from llm_compressor_b200 import (GPTQModifier, Observer, QuantizationModifier, accumulate_hessian_lower,
                                 compress_state_dict, finalize_hessian, make_empty_hessian, oneshot,
                                 preset_name_to_scheme, quantize_weight)
from llm_compressor_b200.awq import scaled_fake_quantize

_DEV = "cuda"


def listed():
    return [
        # the smallest call: one projection of a toy model, where launches and host time are everything
        dict(name="rtn_w4a16_tiny", path="rtn", scheme="W4A16", observer="memoryless_minmax", modules=1, rows=256,
             cols=512),
        # 128 x 128 blocks, the scheme of block-scaled FP8 checkpoints, at an attention projection's size
        dict(name="rtn_fp8_block", path="rtn", scheme="FP8_BLOCK", observer="memoryless_minmax", modules=1, rows=4096,
             cols=4096),
        # gate and up projections of an 8B-sized MLP: one global scale for the two of them
        dict(name="rtn_nvfp4_gate_up", path="rtn", scheme="NVFP4A16", observer="memoryless_minmax", modules=2,
             rows=14336, cols=4096),
        # the grid-search observer on a projection of ordinary size
        dict(name="rtn_w4a16_mse", path="rtn", scheme="W4A16", observer="memoryless_mse", modules=1, rows=4096,
             cols=4096),
        # the scale search behind an input norm: query, key and value projections together
        dict(name="awq_w4a16_qkv", path="awq", scheme="W4A16", modules=3, rows=4096, cols=4096),
        # calibration one short sequence at a time
        dict(name="hessian_short", path="hessian", batches=4, tokens=512, cols=4096),
        # the widest input of an 8B-sized layer over a large batch
        dict(name="hessian_wide", path="hessian", batches=1, tokens=32768, cols=14336),
        # odd sizes, FP8 per channel, columns in order of activation
        dict(name="gptq_fp8_odd", path="gptq", scheme="FP8_DYNAMIC", actorder="static", rows=1001, cols=1160,
             batches=3, tokens=2311),
        # an attention projection, one batch of eight sequences
        dict(name="gptq_w4a16_attn", path="gptq", scheme="W4A16", actorder="", rows=4096, cols=4096, batches=1,
             tokens=16384),
        # the down projection of an 8B-sized MLP: the longest chain of the whole path
        dict(name="gptq_w4a16_down", path="gptq", scheme="W4A16", actorder="", rows=4096, cols=14336, batches=2,
             tokens=28672),
        # a whole decoder layer, hidden 2048 / intermediate 5632, 64 sequences of 512 tokens in batches of 8
        dict(name="layer_w4a16", path="layer", scheme="W4A16", actorder="", experts=0, hidden=2048, inter=5632,
             batches=8, tokens=4096),
        # the experts of a mixture-of-experts layer, every expert calibrated on every token
        dict(name="layer_fp8_experts", path="layer", scheme="FP8_DYNAMIC", actorder="static", experts=32, hidden=2048,
             inter=768, batches=2, tokens=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi, step):
    return max(step, _log(rng, lo, hi) // step * step)


def draw(rng):
    path = rng.choice(["rtn", "rtn", "rtn", "awq", "hessian", "hessian", "gptq", "gptq", "gptq", "layer"])
    if path == "rtn":
        scheme = rng.choice(["W4A16", "W4A16_ASYM", "W8A16", "FP8_DYNAMIC", "FP8_BLOCK", "NVFP4A16", "MXFP4A16",
                             "MXFP8A16"])
        observer = rng.choice(["memoryless_minmax", "memoryless_minmax", "memoryless_mse"])
        modules = 2 if scheme == "NVFP4A16" else 1
        step = {"W4A16": 128, "W4A16_ASYM": 128, "NVFP4A16": 16, "MXFP4A16": 32, "MXFP8A16": 32}.get(scheme, 8)
        most = 4096 if observer == "memoryless_mse" else 14336
        cols = _width(rng, 256, most, step)
        rows = min(_log(rng, 64, most), most * 4096 // cols)
        return dict(path=path, scheme=scheme, observer=observer, modules=modules, rows=rows, cols=cols)
    if path == "awq":
        scheme = rng.choice(["W4A16", "W4A16_ASYM", "W8A16"])
        return dict(path=path, scheme=scheme, modules=rng.choice([1, 2, 3]), rows=_log(rng, 128, 4096),
                    cols=_width(rng, 256, 4096, 128))
    if path == "hessian":
        cols = _width(rng, 256, 14336, 8)
        return dict(path=path, batches=rng.randint(1, 4), tokens=_log(rng, 256, 8192), cols=cols)
    if path == "gptq":
        scheme = rng.choice(["W4A16", "W4A16", "W4A16_ASYM", "W8A16", "FP8_DYNAMIC", "NVFP4A16"])
        step = {"W4A16": 128, "W4A16_ASYM": 128, "NVFP4A16": 16}.get(scheme, 8)
        cols = _width(rng, 256, 8192, step)
        return dict(path=path, scheme=scheme, actorder=rng.choice(["", "static"]), rows=_log(rng, 64, 4096),
                    cols=cols, batches=2, tokens=2 * cols + rng.randint(1, 999))
    if rng.random() < 0.5:
        hidden = _width(rng, 512, 2048, 128)
        return dict(path=path, scheme=rng.choice(["W4A16", "FP8_DYNAMIC"]), actorder=rng.choice(["", "static"]),
                    experts=0, hidden=hidden, inter=min(5632, _width(rng, 2 * hidden, 3 * hidden, 128)),
                    batches=rng.randint(4, 8), tokens=4096)
    return dict(path=path, scheme=rng.choice(["W4A16", "FP8_DYNAMIC"]), actorder=rng.choice(["", "static"]),
                experts=rng.randint(16, 32), hidden=_width(rng, 512, 2048, 128), inter=_width(rng, 256, 768, 128),
                batches=2, tokens=rng.randint(3072, 4096))


# ---------------------------------------------------------------------------------------- inputs
def _weight(g, rows, cols, outliers=False):
    w = torch.randn(rows, cols, generator=g, device=_DEV) * 0.02
    if outliers:
        rare = torch.rand(rows, cols, generator=g, device=_DEV) < 1e-3
        w = torch.where(rare, 25.0 * w, w)
    return w.to(torch.bfloat16)


def _linear(weight):
    lin = torch.nn.Linear(weight.shape[1], weight.shape[0], bias=False, device="meta", dtype=weight.dtype)
    lin.weight = torch.nn.Parameter(weight, requires_grad=False)
    return lin


def _activations(g, tokens, cols):
    """[1, tokens, cols]: channels differ in scale by up to a factor of nine."""
    scale = 0.25 + 2.0 * torch.rand(cols, generator=g, device=_DEV)
    x = torch.empty(1, tokens, cols, dtype=torch.bfloat16, device=_DEV)
    for t in range(0, tokens, 8192):
        part = x[0, t:t + 8192]
        part.copy_(torch.randn(part.shape, generator=g, device=_DEV) * scale)
    return x


def _siblings(case, g, outliers):
    """Linear modules of one parent, named as the siblings that share a global scale are."""
    names = {1: ["o_proj"], 2: ["gate_proj", "up_proj"], 3: ["q_proj", "k_proj", "v_proj"]}[case["modules"]]
    model = torch.nn.Module()
    for name in names:
        model.add_module(name, _linear(_weight(g, case["rows"], case["cols"], outliers)))
    return model


def _decoder_modules(case, g):
    """(parent, [(name, module, input name)]) of a decoder layer's projections, 4 query heads to a KV head."""
    h, i = case["hidden"], case["inter"]
    rows = [("q_proj", h, "attn"), ("k_proj", h // 4, "attn"), ("v_proj", h // 4, "attn"), ("o_proj", h, "out"),
            ("gate_proj", i, "mlp"), ("up_proj", i, "mlp"), ("down_proj", h, "down")]
    parent, mods = torch.nn.Module(), []
    for name, n, key in rows:
        lin = _linear(_weight(g, n, i if key == "down" else h))
        parent.add_module(name, lin)
        mods.append((name, lin, key))
    return parent, mods, {"attn": h, "out": h, "mlp": h, "down": i}


def _expert_modules(case, g):
    """The experts' projections, cut out of one [experts, rows, cols] tensor per kind as checkpoints store them."""
    e, h, i = case["experts"], case["hidden"], case["inter"]
    parent, mods, stacks = torch.nn.Module(), [], {}
    for kind, n, k in (("gate_proj", i, h), ("up_proj", i, h), ("down_proj", h, i)):
        stacks[kind] = _weight(g, e * n, k).view(e, n, k)
    for j in range(e):
        for kind, stack in stacks.items():
            lin = _linear(stack[j])
            parent.add_module("expert_%d_%s" % (j, kind), lin)
            mods.append(("expert_%d_%s" % (j, kind), lin, "mlp" if kind != "down_proj" else "down_%d" % j))
    return parent, mods, dict({"mlp": h}, **{"down_%d" % j: i for j in range(e)}), stacks


def prepare(case, seed):
    g = torch.Generator(device=_DEV).manual_seed(seed)
    s = {"case": case, "path": case["path"]}
    if case["path"] == "rtn":
        s["model"] = _siblings(case, g, True)
    elif case["path"] == "awq":
        s["model"] = _siblings(case, g, False)
        s["layers"] = list(s["model"].children())
        for lin in s["layers"]:
            lin.quantization_scheme = preset_name_to_scheme(case["scheme"], ["Linear"])
        s["weights"] = [lin.weight.data.clone() for lin in s["layers"]]
        s["scales"] = torch.exp(0.5 * torch.randn(case["cols"], generator=g, device=_DEV))
    elif case["path"] in ("hessian", "gptq"):
        s["module"] = _linear(_weight(g, case.get("rows", 8), case["cols"]))
        s["batches"] = [_activations(g, case["tokens"], case["cols"]) for _ in range(case["batches"])]
        if case["path"] == "gptq":
            scheme = preset_name_to_scheme(case["scheme"], ["Linear"])
            # act-order "static" is also meant for per-channel schemes, as the modifier sets it
            object.__setattr__(scheme.weights, "actorder", "weight" if case["actorder"] else None)
            s["scheme"] = scheme
    else:
        if case["experts"]:
            parent, mods, widths, stacks = _expert_modules(case, g)
            s["stacks"] = stacks
            s["given"] = {k: v.clone() for k, v in stacks.items()}
        else:
            parent, mods, widths = _decoder_modules(case, g)
            s["given"] = {name: lin.weight.data.clone() for name, lin, _ in mods}
        s["parent"], s["mods"] = parent, mods
        s["inputs"] = [{key: _activations(g, case["tokens"], k) for key, k in widths.items()}
                       for _ in range(case["batches"])]
    return s


# ------------------------------------------------------------------------------------- one pass
def _run_rtn(s):
    case, model = s["case"], s["model"]
    oneshot(model, recipe=QuantizationModifier(targets="Linear", scheme=case["scheme"],
                                               weight_observer=case["observer"]))
    out = {}
    for name, lin in model.named_children():
        state = {"weight": lin.weight.data, "weight_scale": lin.weight_scale.data,
                 "weight_zero_point": lin.weight_zero_point.data}
        if hasattr(lin, "weight_global_scale"):
            state["weight_global_scale"] = lin.weight_global_scale.data
        out[name] = compress_state_dict(state, lin.quantization_scheme)
    return out


def _run_hessian(s):
    H, n = make_empty_hessian(s["module"]), 0
    for x in s["batches"]:
        H, n = accumulate_hessian_lower(x, H, n)
    return finalize_hessian(H, n)


def _run_gptq(s):
    lin, scheme = s["module"], s["scheme"]
    H = _run_hessian(s)
    lin.weight_observer = Observer.load_from_registry("memoryless_minmax", base_name="weight", args=scheme.weights)
    loss, out = quantize_weight(lin, scheme.weights, H)
    return {"loss": loss, "weight": out["weight"], "stored": compress_state_dict(out, scheme)}


def _run_layer(s):
    case, parent = s["case"], s["parent"]
    # the weights as the checkpoint holds them: the pass before this one has quantised them in place
    if case["experts"]:
        for kind, stack in s["stacks"].items():
            stack.copy_(s["given"][kind])
    else:
        for name, lin, _ in s["mods"]:
            lin.weight.data.copy_(s["given"][name])
    mod = GPTQModifier(targets="Linear", scheme=case["scheme"], actorder=case["actorder"] or None)
    mod.on_initialize(parent)
    mod.on_calibration_start(parent)
    for inputs in s["inputs"]:
        for _, lin, key in s["mods"]:
            mod.calibrate_module(lin, (inputs[key],), None)
    mod.on_sequential_epoch_end(parent, list(parent.modules()))
    mod.on_calibration_end(parent)
    mod.on_finalize(parent)
    scales = torch.cat([lin.weight_scale.data.reshape(-1) for _, lin, _ in s["mods"]])
    weights = dict(s["stacks"]) if case["experts"] else {name: lin.weight.data for name, lin, _ in s["mods"]}
    return {"scales": scales, "losses": list(mod.losses.values())[:32], "weights": weights}


def run(state):
    path = state["path"]
    if path == "rtn":
        return _run_rtn(state)
    if path == "awq":
        return scaled_fake_quantize(state["weights"], state["scales"], state["layers"], state["model"])
    if path == "hessian":
        return _run_hessian(state)
    if path == "gptq":
        return _run_gptq(state)
    return _run_layer(state)


# ------------------------------------------------------------------------------ least work of a pass
def _code_bytes(scheme):
    """(bytes of a stored code, elements to a stored scale or 0 for one per row or block)"""
    return {"W4A16": (0.5, 128), "W4A16_ASYM": (0.5, 128), "NVFP4A16": (0.5, 16), "MXFP4A16": (0.5, 32),
            "MXFP8A16": (1.0, 32)}.get(scheme, (1.0, 0))


def _solve(rows, cols):
    """Factorisation of one Hessian is 2/3 K^3; the sweep of one weight N K^2."""
    return 2.0 * cols ** 3 / 3.0, float(rows) * cols * cols


def work(case):
    path = case["path"]
    if path in ("rtn", "awq"):
        n = float(case["modules"]) * case["rows"] * case["cols"]
        code, group = _code_bytes(case["scheme"])
        if path == "awq":
            return {"bytes": 4.0 * n, "flops": 4.0 * n}
        # twenty candidates of the grid search, about four operations each on every element
        ops = 80.0 if case["observer"] == "memoryless_mse" else 4.0
        return {"bytes": n * (2.0 + code + (2.0 / group if group else 0.0)), "flops": ops * n}
    if path in ("hessian", "gptq"):
        t, k = float(case["batches"]) * case["tokens"], case["cols"]
        b, f = 2.0 * t * k, t * k * (k + 1)
        if path == "hessian":
            return {"bytes": b + 4.0 * k * k, "flops": f}
        factor, sweep = _solve(case["rows"], k)
        return {"bytes": b + case["rows"] * k * (4.0 + _code_bytes(case["scheme"])[0]), "flops": f + factor + sweep}
    t, h, i, e = float(case["batches"]) * case["tokens"], case["hidden"], case["inter"], case["experts"]
    if e:
        shapes, widths = [(2 * e * i, h), (e * h, i)], [h] + [i] * e
        weights = 3.0 * e * h * i
    else:
        shapes, widths = [(2 * h + h // 2, h), (2 * i, h), (h, i)], [h, h, h, i]
        weights = 2.5 * h * h + 3.0 * h * i
    flops = sum(t * k * (k + 1) + _solve(0, k)[0] for k in widths) + sum(_solve(n, k)[1] for n, k in shapes)
    return {"bytes": 2.0 * t * sum(widths) + 4.0 * weights, "flops": flops}


def tolerance(case):
    path = case["path"]
    if path == "awq" or (path == "rtn" and case["observer"] == "memoryless_minmax"):
        return "exact"
    if path == "rtn":
        # the search compares float32 sums of errors: where two candidates are equal to rounding, either may win
        return {"rel": 5e-3, "max": 0.3, "differ": 5e-3}
    if path == "hessian":
        return {"rel": 1e-4, "max": 1e-3}
    # float32 sums of another order turn a few codes at rounding boundaries; one step of a 4-bit code is up to
    # about 0.9 of the weights' root mean square
    return {"rel": 1e-2, "max": 0.95, "differ": 8e-3}
