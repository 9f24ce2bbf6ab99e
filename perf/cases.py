"""The calls whose speed this framework is judged by, over the sizes, types and options that a program built on it meets.

A program holds weights, activations and caches on the GPU and calls the backend (``torchlette_b200.backend``) on them: packed-weight
products of a decode step and of a prefill, dense products, attention over a KV cache, a whole decoder layer through the op API, the
quantizer that a loader runs, and a full stack of decode projections replayed as one graph.  Buffers here are torch tensors that the
backend's ``CudaTensor`` wraps; the calls are the public ones.

A case is a dict of plain values.  ``listed`` names the representative ones, ``draw`` makes another of the same ranges.
"""
import math

import torch

from torchlette_b200 import CudaTensor, EpilogueConfig, getBackend, perChannelFormat, resolveWeightFormat
from torchlette_b200.decode_stack import DecodeStack, StackConfig

_TORCH = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "u32": torch.int32, "u16": torch.int16}
_SIZE = {"f32": 4, "f16": 2, "bf16": 2}
_DEV = "cuda"


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------

def _linear(name, m, n, k, fmt, act, out, epilogue, layout="nt"):
    return {"name": name, "kind": "linear", "m": m, "n": n, "k": k, "format": fmt, "act": act, "out": out, "epilogue": epilogue,
            "layout": layout}


def listed():
    return [
        # the smallest call of a decode step: one q projection of a 0.6B-shaped model for one token; latency and host path count
        _linear("decode_small_m1", 1, 2048, 1024, "int8-channel", "f16", "f16", "none"),
        # one token through a packed weight with f32 activations, the type torchlette's own frontend computes in by default, in its
        # default weight format
        _linear("decode_f32_m1_int8_64", 1, 4096, 4096, "int8-64", "f32", "f32", "none"),
        # small-batch decode through the MLP's wide projection with bias and gelu fused, sixteen sequences
        _linear("decode_mlp_m16", 16, 14336, 4096, "int8-channel", "f16", "f16", "bias+gelu"),
        # the same projection with int4 weights, four sequences
        _linear("decode_int4_m4", 4, 14336, 4096, "int4-128", "f16", "f16", "bias+gelu"),
        # a prompt of an odd length through the gate projection, weights in the default grouped format
        _linear("prefill_ragged_int8_64", 333, 12288, 4096, "int8-64", "f16", "f16", "silu"),
        # a long prompt (or several together) through the MLP on the tensor cores
        _linear("prefill_mlp_2048", 2048, 14336, 4096, "int8-channel", "bf16", "bf16", "gelu"),
        # an unquantized linear layer on an odd number of tokens
        _linear("dense_linear_1000", 1000, 4096, 4096, "dense", "bf16", "bf16", "bias+gelu"),
        # one new token per sequence against a filled KV cache, grouped query heads
        {"name": "attention_decode", "kind": "attention", "batch": 8, "heads": 32, "kv_heads": 8, "dim": 128, "q_len": 1, "kv_len": 4000,
         "dtype": "f16"},
        # the prompt's own causal attention
        {"name": "attention_prefill", "kind": "attention", "batch": 1, "heads": 32, "kv_heads": 8, "dim": 128, "q_len": 2048,
         "kv_len": 2048, "dtype": "f16"},
        # one token per sequence through a whole 8B-shaped decoder layer, op by op as an eager program writes it
        {"name": "decoder_layer_step", "kind": "layer", "batch": 2, "hidden": 4096, "heads": 32, "kv_heads": 8, "dim": 128, "inter": 12288,
         "kv_len": 700, "dtype": "f16"},
        # loading a weight: f32 on the device to packed int8 and its scales
        {"name": "quantize_load", "kind": "quantize", "n": 12288, "k": 4096, "format": "int8-64"},
        # all weight products of a decode step of an 8B-shaped model at batch 8, one replayed graph (the headline workload)
        {"name": "decode_stack_m8", "kind": "stack", "layers": 36, "batch": 8, "hidden": 4096, "kv_out": 1024, "inter": 12288,
         "vocab": 151936, "act": "f16"},
    ]


def _between(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "int4", "prefill", "prefill", "dense", "attention", "attention", "layer", "quantize",
                       "stack"])
    if kind in ("decode", "int4", "prefill", "dense"):
        k = _between(rng, 512, 14336, 128)
        n = _between(rng, 512, min(151936, 14336 * 4096 // k), rng.choice([1, 8, 64, 64]))
        act = rng.choice(["f16", "f16", "bf16", "f32"]) if kind == "decode" else rng.choice(["f16", "bf16"])
        out = rng.choice([act, act, "f32"])
        epilogue = rng.choice(["none", "none", "bias+gelu", "silu", "bias+relu"])
        if kind == "decode":
            return _linear("", rng.choice([1, 1, 2, 3, 4, 8, 8, 13, 16]), n, k, rng.choice(["int8-channel", "int8-64", "int8-64", "int8-128"]),
                           act, out, epilogue)
        if kind == "int4":
            return _linear("", rng.choice([1, 1, 4, 8, 16]), n, k, rng.choice(["int4-128", "int4-128", "int4-32"]), act, out, epilogue)
        m = _between(rng, 17, 2048)
        if kind == "prefill":
            return _linear("", m, n, k, rng.choice(["int8-channel", "int8-64", "int8-64", "int8-128", "int4-128"]), act, out, epilogue)
        n = max(512, n // 8 * 8)
        return _linear("", m, n, k, "dense", act, out, epilogue, rng.choice(["nt", "nt", "nn"]))
    if kind == "attention":
        heads, kv_heads = rng.choice([(32, 8), (32, 8), (16, 8), (16, 4), (8, 8)])
        case = {"kind": "attention", "heads": heads, "kv_heads": kv_heads, "dim": rng.choice([64, 128, 128]),
                "dtype": rng.choice(["f16", "f16", "bf16"])}
        if rng.random() < 0.5:
            return dict(case, batch=rng.choice([1, 2, 4, 8]), q_len=1, kv_len=_between(rng, 40, 4000))
        q_len = _between(rng, 30, 2048)
        # a prompt on its own, or a chunk of one behind what the cache already holds
        return dict(case, batch=1, q_len=q_len, kv_len=q_len if rng.random() < 0.7 else _between(rng, q_len, 2048))
    if kind == "layer":
        hidden = rng.choice([1024, 2048, 4096])
        return {"kind": "layer", "batch": rng.choice([1, 2, 4, 8]), "hidden": hidden, "heads": hidden // 128, "kv_heads": min(8, hidden // 128),
                "dim": 128, "inter": hidden * 3, "kv_len": _between(rng, 40, 2000), "dtype": rng.choice(["f16", "f16", "f32"])}
    if kind == "quantize":
        k = _between(rng, 512, 12288, 128)
        return {"kind": "quantize", "n": _between(rng, 500, 12288 * 4096 // k), "k": k, "format": rng.choice(["int8-64", "int8-64", "int8-128"])}
    hidden = rng.choice([1024, 2048, 4096])
    act = rng.choice(["f16", "f16", "bf16"])
    return {"kind": "stack", "layers": _between(rng, 2, 30 if act == "f16" else 7), "batch": rng.choice([1, 2, 4, 8]), "hidden": hidden,
            "kv_out": 1024, "inter": hidden * 3, "vocab": rng.choice([32000, 50304, 151936]), "act": act}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device=_DEV).manual_seed(int(seed))


def _normal(gen, shape, dtype="f32", scale=1.0):
    return (torch.randn(*shape, device=_DEV, generator=gen) * scale).to(_TORCH[dtype])


def _wrap(t, dtype, shape=None, **more):
    return CudaTensor(getBackend(), list(shape if shape is not None else t.shape), dtype, t.data_ptr(), t.numel() * t.element_size(),
                      ownsBuffer=False, **more)


def _format(name, k):
    return perChannelFormat(k) if name == "int8-channel" else resolveWeightFormat(name)


def _weight(gen, n, k, fmt):
    """A packed [n, k] weight: random int8 with per-channel f32 scales, or a normal matrix quantized in groups with f16 scales."""
    storage = _format(fmt, k)
    if fmt == "int8-channel":
        q = torch.randint(-127, 128, (n, k), dtype=torch.int8, device=_DEV, generator=gen)
        scales = torch.empty(n, 1, device=_DEV).uniform_(0.001, 0.01, generator=gen)
        scales_dtype = "f32"
    else:
        group, top = storage.packing.groupSize, (127 if fmt.startswith("int8") else 7)
        w = torch.randn(n, k // group, group, device=_DEV, generator=gen).mul_(1.0 / math.sqrt(k))
        scales = w.abs().amax(2).to(torch.float16)
        q = w.mul_(top / scales.float().unsqueeze(2)).add_(0.5).floor_().clamp_(-top, top).to(torch.int8).reshape(n, k)
        scales_dtype = "u16"
        if top == 7:
            nib = (q & 15).view(n, k // 2, 2)
            q = nib[:, :, 0] | (nib[:, :, 1] << 4)  # two nibbles a byte, eight a word, the lowest k in the lowest bits
    q = q.contiguous()
    return _wrap(q, "f16", [n, k], format=storage, scales=_wrap(scales, scales_dtype)), (q, scales)


def _epilogue(case, gen):
    ops, inputs, keep = [], [], []
    for part in case["epilogue"].split("+"):
        if part == "bias":
            bias = _normal(gen, (case["n"],), scale=0.02)
            keep.append(bias)
            inputs.append(_wrap(bias, "f32"))
            ops.append({"kind": "bias", "inputIndex": 0})
        elif part != "none":
            ops.append({"kind": "unary", "op": part})
    return {"epilogue": EpilogueConfig(ops, len(inputs), case["out"]), "epilogueInputs": inputs}, keep


def _prepare_linear(case, gen):
    m, n, k = case["m"], case["n"], case["k"]
    ops = getBackend().ops
    x = _normal(gen, (m, k), case["act"])
    y = torch.empty(m, n, device=_DEV, dtype=_TORCH[case["out"]])
    if case["format"] == "dense":
        w = _normal(gen, (n, k) if case["layout"] == "nt" else (k, n), case["act"], 1.0 / math.sqrt(k))
        keep, b = (w,), _wrap(w, case["act"])
        b = ops.transpose(b) if case["layout"] == "nt" else b
    else:
        weight, keep = _weight(gen, n, k, case["format"])
        b = ops.transpose(weight)
    options, more = _epilogue(case, gen)
    if case["format"] == "int8-channel":
        options["alpha"] = 1.0 / (0.44 * math.sqrt(k))  # keeps the products of the random integers near one
    options["outBuffer"] = _wrap(y, case["out"])
    return {"x": _wrap(x, case["act"]), "b": b, "options": options, "y": y, "keep": (x, keep, more)}


def _prepare_attention(case, gen):
    b, h, g, d, s, n = (case[f] for f in ("batch", "heads", "kv_heads", "dim", "q_len", "kv_len"))
    capacity = (n + 255) // 256 * 256
    q = _normal(gen, (b, h, s, d), case["dtype"])
    k, v = _normal(gen, (b, g, capacity, d), case["dtype"]), _normal(gen, (b, g, capacity, d), case["dtype"])
    return {"q": _wrap(q, case["dtype"]), "k": _wrap(k, case["dtype"]), "v": _wrap(v, case["dtype"]), "kv_len": n,
            "scale": 1.0 / math.sqrt(d), "one": s == 1, "out": None, "keep": (q, k, v)}


def _prepare_layer(case, gen):
    hidden, h, g, d, inter, dt = (case[f] for f in ("hidden", "heads", "kv_heads", "dim", "inter", "dtype"))
    b, capacity, pos = case["batch"], (case["kv_len"] + 255) // 256 * 256, case["kv_len"] - 1
    state = {"keep": [], "pos": pos, "case": dict(case), "out": None}
    for name, n, k in (("q", h * d, hidden), ("k", g * d, hidden), ("v", g * d, hidden), ("o", hidden, h * d), ("gate", inter, hidden),
                       ("up", inter, hidden), ("down", hidden, inter)):
        state[name], keep = _weight(gen, n, k, "int8-64")
        state["keep"].append(keep)
    angle = torch.arange(capacity, device=_DEV).unsqueeze(1) / 1e6 ** (torch.arange(d // 2, device=_DEV) / (d // 2))
    for name, t, dtype in (("n_in", 1 + _normal(gen, (hidden,), scale=0.2), "f32"), ("n_post", 1 + _normal(gen, (hidden,), scale=0.2), "f32"),
                           ("n_q", 1 + _normal(gen, (d,), scale=0.2), "f32"), ("n_k", 1 + _normal(gen, (d,), scale=0.2), "f32"),
                           ("cos", angle.cos(), "f32"), ("sin", angle.sin(), "f32"), ("x", _normal(gen, (b, hidden), dt), dt),
                           ("k_cache", _normal(gen, (b, g, capacity, d), dt), dt), ("v_cache", _normal(gen, (b, g, capacity, d), dt), dt)):
        t = t.contiguous()
        state[name] = _wrap(t, dtype)
        state["keep"].append(t)
        if name.endswith("cache"):
            state[name + "_t"] = t
    return state


def _prepare_quantize(case, gen):
    w = _normal(gen, (case["n"], case["k"]), scale=0.02)
    return {"w": _wrap(w, "f32"), "format": resolveWeightFormat(case["format"]), "out": None, "keep": w}


class _Stack(DecodeStack):
    """A stack that gives its graph back when the program drops it."""

    def __del__(self):
        self.destroy()


def _prepare_stack(case, gen, seed):
    cfg = StackConfig(hidden=case["hidden"], layers=case["layers"], q_out=case["hidden"], kv_out=case["kv_out"], inter=case["inter"],
                      vocab=case["vocab"], batch=case["batch"], act_dtype=case["act"])
    stack = _Stack(getBackend(), cfg, seed=int(seed) * 100_003)
    stack.x.copy_(_normal(gen, (case["batch"], case["hidden"]), case["act"]))
    torch.cuda.synchronize()
    stack.capture()
    return {"stack": stack}


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "stack":
        state = _prepare_stack(case, gen, seed)
    else:
        state = {"linear": _prepare_linear, "attention": _prepare_attention, "layer": _prepare_layer, "quantize": _prepare_quantize}[kind](case, gen)
    state["kind"] = kind
    torch.cuda.synchronize()  # the backend has a stream of its own
    return state


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

class _Memory:
    def __init__(self, ptr, shape, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "typestr": typestr, "version": 2}


def _view(t, dtype=None):
    """A backend tensor's memory as a torch tensor (no copy; bf16 as its 16 bits)."""
    typestr = {"f32": "<f4", "f16": "<f2", "bf16": "<i2", "u32": "<i4", "u16": "<i2"}[dtype or t.dtype]
    return torch.as_tensor(_Memory(t.buffer, t.shape, typestr), device=_DEV)


def _drop(state):
    """The last pass's result goes before the next is made, as a program's temporaries do."""
    last, state["out"] = state["out"], None
    for t in last or ():
        t.destroy()


def _run_layer(state):
    be, case, pos = getBackend(), state["case"], state["pos"]
    ops, b, h, g, d, dt = be.ops, case["batch"], case["heads"], case["kv_heads"], case["dim"], case["dtype"]
    h0 = ops.rmsnorm(state["x"], state["n_in"], 1e-6)
    q, k, v = (be.linear(h0, state[w], None, None, dt) for w in ("q", "k", "v"))
    qn = ops.rmsnorm(ops.reshape(q, [b, h, d]), state["n_q"], 1e-6)
    kn = ops.rmsnorm(ops.reshape(k, [b, g, d]), state["n_k"], 1e-6)
    at = {"cosOffset": pos * (d // 2), "sinOffset": pos * (d // 2)}
    qr = ops.fusedRoPE(ops.reshape(qn, [b, h, 1, d]), state["cos"], state["sin"], at)
    kr = ops.fusedRoPE(ops.reshape(kn, [b, g, 1, d]), state["cos"], state["sin"], at)
    ops.kvAppend(state["k_cache"], kr, pos)
    ops.kvAppend(state["v_cache"], v, pos)
    attn = ops.decodeAttention(qr, state["k_cache"], state["v_cache"], pos + 1, 1.0 / math.sqrt(d))
    o = be.linear(ops.reshape(attn, [b, h * d]), state["o"], None, None, dt)
    h1 = ops.add(state["x"], o)
    h1n = ops.rmsnorm(h1, state["n_post"], 1e-6)
    gu = be.swiglu(h1n, state["gate"], state["up"], dt)
    down = be.linear(gu, state["down"], None, None, dt)
    out = ops.add(h1, down)
    for t in (h0, q, k, v, qn, kn, qr, kr, attn, o, h1, h1n, gu, down):
        t.destroy()
    return out


def run(state):
    be, kind = getBackend(), state["kind"]
    if kind == "linear":
        be.ops.matmul(state["x"], state["b"], state["options"])
        return state["y"]
    if kind == "stack":
        stack = state["stack"]
        stack.step()
        return {"logits": stack.logits, "hidden": stack.h2}
    _drop(state)
    if kind == "attention":
        if state["one"]:
            out = be.ops.decodeAttention(state["q"], state["k"], state["v"], state["kv_len"], state["scale"])
        else:
            out = be.ops.attention(state["q"], state["k"], state["v"], state["kv_len"], state["scale"], causal=True)
        state["out"] = (out,)
        y = _view(out)
        return y.view(torch.bfloat16) if out.dtype == "bf16" else y
    if kind == "layer":
        out = _run_layer(state)
        state["out"] = (out,)
        return {"hidden": _view(out), "k_cache": state["k_cache_t"], "v_cache": state["v_cache_t"]}
    w = be.quantizeLinearWeightOnDevice(state["w"], state["format"])
    state["out"] = (w, w.scales)
    n, k = w.shape
    packed = torch.as_tensor(_Memory(w.buffer, (n, k // 4), "<i4"), device=_DEV)
    return {"packed": packed, "scales": _view(w.scales)}


# ---------------------------------------------------------------------------
# What a pass cannot do without, and how far two correct results may be apart
# ---------------------------------------------------------------------------

def _weight_bytes(n, k, fmt, act="f16"):
    if fmt == "dense":
        return n * k * _SIZE[act]
    if fmt == "int8-channel":
        return n * k + 4 * n
    packing = resolveWeightFormat(fmt).packing
    return n * k // (1 if packing.scheme == "int8-grouped" else 2) + 2 * n * (k // packing.groupSize)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        bias = 4 * n if "bias" in case["epilogue"] else 0
        return {"bytes": _weight_bytes(n, k, case["format"], case["act"]) + m * k * _SIZE[case["act"]] + m * n * _SIZE[case["out"]] + bias,
                "flops": 2 * m * n * k}
    if kind == "attention":
        b, h, g, d, s, n = (case[f] for f in ("batch", "heads", "kv_heads", "dim", "q_len", "kv_len"))
        pairs = s * n - s * (s - 1) // 2 if s > 1 else n  # query s sees the keys up to its own position
        return {"bytes": b * d * _SIZE[case["dtype"]] * (2 * h * s + 2 * g * n), "flops": 4 * b * h * d * pairs}
    if kind == "layer":
        b, h, g, d, hidden, inter, n = (case[f] for f in ("batch", "heads", "kv_heads", "dim", "hidden", "inter", "kv_len"))
        weights = [(h * d, hidden), (g * d, hidden), (g * d, hidden), (hidden, h * d), (inter, hidden), (inter, hidden), (hidden, inter)]
        size = _SIZE[case["dtype"]]
        return {"bytes": sum(_weight_bytes(r, c, "int8-64") for r, c in weights) + b * size * (2 * hidden + 2 * g * d * n) + 4 * (2 * hidden + 3 * d),
                "flops": sum(2 * b * r * c for r, c in weights) + 4 * b * h * d * n}
    if kind == "quantize":
        n, k = case["n"], case["k"]
        return {"bytes": 4 * n * k + _weight_bytes(n, k, case["format"]), "flops": 2 * n * k}
    cfg = StackConfig(hidden=case["hidden"], layers=case["layers"], q_out=case["hidden"], kv_out=case["kv_out"], inter=case["inter"],
                      vocab=case["vocab"], batch=case["batch"], act_dtype=case["act"])
    return {"bytes": cfg.algorithmic_bytes_per_step(), "flops": cfg.flops_per_step()}


def tolerance(case):
    """About four times what each path differs by from itself in 64 bits (products, attention) or with its sums in another order (layer,
    stack): one rounding to f16 is 2.1e-4 of the result, one to bf16 1.7e-3, f32 sums 1.3e-7 and the tensor cores' f32 sums up to 1.4e-5."""
    kind = case["kind"]
    rounding = {"f16": 9e-4, "bf16": 7e-3, "f32": 5e-6}
    if kind == "linear":
        own = rounding[case["out"]]
        if case["m"] > 16:
            own = max(own, 6e-5)
            if case["format"] not in ("dense", "int8-channel"):  # the dequantized weight is an operand of the activations' type
                own = {"f16": 1.3e-3, "bf16": 1e-2}[case["act"]]
        return {"rel": own}
    if kind == "attention":
        return {"rel": rounding[case["dtype"]]}
    if kind == "layer":
        return {"rel": {"f16": 1e-3, "f32": 5e-6}[case["dtype"]]}
    if kind == "quantize":
        return "exact"
    # every layer's hand-over is rounded to the activation type and nothing is normalised between layers, so a last bit grows with depth
    rel = {"f16": 1.2e-3, "bf16": 4e-3}[case["act"]] * case["layers"]
    return {"rel": min(0.03, rel), "max": min(0.4, 14 * rel)}
