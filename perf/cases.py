"""Performance cases: the work that programs using this package have it do, through its public entry points.

A case is one *pass* of one of three operations:

``products``    ``matmul(x, w)`` for every weight of the case: one weight, or the seven weights of a decoder
                layer (q, k, v, o, gate, up, down), each output kept.  ``m`` is the flattened batch: 1 for
                generation, a few up to 32 for batched decoding and speculative checks, hundreds for chunked
                prefill, thousands for prefill of whole prompts.
``train``       the same product with a gradient in ``x`` (the package's frozen-weight training step): the
                forward result and ``dx``.
``dequantize``  ``QuantizedArray.dequantize(dtype)``: a dense copy of the weight.

Weights are random block bytes with small finite scales, activations N(0, 1) in bfloat16: what the formats hold and
what a norm layer hands to a linear layer.
"""
import concurrent.futures
import math

import numpy as np
import torch

import gguf_jax_b200 as gj
from gguf_jax_b200 import quants as _quants
from gguf_jax_b200 import synth

QT = gj.GGMLQuantizationType
_gguf = _quants._ref            # the third-party numpy decoder (gguf.quants): the definition of every format
_K_QUANTS = ("Q4_K", "Q5_K", "Q6_K")
_LOWBIT = ("Q2_K", "Q3_K", "IQ1_S", "IQ1_M", "IQ2_XXS", "IQ2_XS", "IQ2_S", "IQ3_XXS", "IQ3_S", "IQ4_XS", "TQ1_0", "TQ2_0")
_LEGACY = ("Q4_0", "Q4_1", "Q5_0", "Q5_1", "Q8_0", "IQ4_NL", "MXFP4", "NVFP4")
_MAX_WEIGHTS = 28672 * 8192     # largest weight of the listed cases
_MAX_MACS = _MAX_WEIGHTS * 2048


def _layer(name, hidden, kv, inter, attn, v, mlp, down, m):
    return {"name": name, "op": "products", "layer": True, "hidden": hidden, "kv": kv, "inter": inter,
            "attn": attn, "v": v, "mlp": mlp, "down": down, "m": m}


def _single(name, op, qtype, n, k, m, dtype="bfloat16"):
    return {"name": name, "op": op, "layer": False, "qtype": qtype, "n": n, "k": k, "m": m, "dtype": dtype}


def listed():
    return [
        # one token through the linear layers of a small (1B-shaped) Q4_K_M decoder layer: seven short calls, where
        # launches and the host path count
        _layer("decode_1b_layer_m1", 2048, 512, 8192, "Q4_K", "Q6_K", "Q4_K", "Q6_K", 1),
        # the same layer for eight concurrent sequences
        _layer("decode_1b_layer_m8", 2048, 512, 8192, "Q4_K", "Q6_K", "Q4_K", "Q6_K", 8),
        # one token through the largest Q4_K weight of a 70B-shaped layer: the memory-bound headline product
        _single("decode_70b_q4_k_m1", "products", "Q4_K", 8192, 28672, 1),
        # 32 concurrent sequences through an 8B-shaped layer, Q5_K attention and Q6_K feed-forward
        _layer("decode_8b_layer_m32", 4096, 1024, 14336, "Q5_K", "Q5_K", "Q6_K", "Q6_K", 32),
        # a 512-token prefill chunk through the same layer
        _layer("prefill_8b_layer_m512", 4096, 1024, 14336, "Q5_K", "Q5_K", "Q6_K", "Q6_K", 512),
        # a 2048-token prompt through a 70B-shaped gate projection: the largest product
        _single("prefill_70b_q4_k_m2048", "products", "Q4_K", 28672, 8192, 2048),
        # generation with 2-bit code-book weights (70B-shaped, the way such a model fits a small memory)
        _single("lowbit_iq2_xs_m1", "products", "IQ2_XS", 8192, 28672, 1),
        # batched generation with 3-bit code-book weights
        _single("lowbit_iq3_s_m8", "products", "IQ3_S", 8192, 28672, 8),
        # generation with 8-bit legacy blocks (8B-shaped gate projection)
        _single("legacy_q8_0_m1", "products", "Q8_0", 14336, 4096, 1),
        # a few sequences through a weight whose rows are neither 16-byte aligned nor a multiple of any tile
        _single("ragged_q6_k_m5", "products", "Q6_K", 5003, 11 * 256, 5),
        # a dense bf16 copy of a 70B-shaped weight (conversion, merging, frameworks that want dense weights)
        _single("dequantize_q4_k", "dequantize", "Q4_K", 28672, 8192, 0),
        # fine-tuning with frozen quantized weights: forward and input gradient of 1024 tokens
        _single("train_8b_q6_k_m1024", "train", "Q6_K", 14336, 4096, 1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_mult(rng, lo, hi, step):
    return step * max(1, _log_int(rng, lo, hi) // step)


def draw(rng):
    kind = rng.choice(["layer", "decode", "decode", "decode", "batch", "prefill", "train", "dequantize"])
    if kind == "layer":
        hidden = _log_mult(rng, 1024, 5120, 256)
        c = _layer(None, hidden, _log_mult(rng, 256, 1024, 64), _log_mult(rng, 2 * hidden, 4 * hidden, 256),
                   rng.choice(_K_QUANTS), rng.choice(_K_QUANTS), rng.choice(_K_QUANTS), rng.choice(_K_QUANTS), _log_int(rng, 1, 512))
    else:
        family = rng.choice([_K_QUANTS, _K_QUANTS, _LOWBIT, _LEGACY])
        qtype = rng.choice(family)
        k = _log_mult(rng, 1024, 28672, 32 * rng.choice([1, 8]) if family is _LEGACY and qtype != "NVFP4" else 256)
        n = _log_int(rng, 500, 28672)
        if rng.random() < 0.5:
            n = max(256, n // 256 * 256)
        n = min(n, _MAX_WEIGHTS // k)
        m = {"decode": 1 if rng.random() < 0.5 else _log_int(rng, 2, 16), "batch": _log_int(rng, 17, 512),
             "prefill": _log_int(rng, 512, 2048), "train": _log_int(rng, 128, 1024), "dequantize": 0}[kind]
        dtype = rng.choice(["bfloat16", "float32", "float16"]) if kind == "dequantize" else "bfloat16"
        c = _single(None, kind if kind in ("train", "dequantize") else "products", qtype, n, k, m, dtype)
    del c["name"]
    return c


def _weights(case):
    """(label, qtype name, rows, columns, which activation) of every product of the case."""
    if not case["layer"]:
        return [("w", case["qtype"], case["n"], case["k"], "x")]
    h, kv, inter = case["hidden"], case["kv"], case["inter"]
    return [("q", case["attn"], h, h, "attn_in"), ("k", case["attn"], kv, h, "attn_in"), ("v", case["v"], kv, h, "attn_in"),
            ("o", case["attn"], h, h, "attn_out"), ("gate", case["mlp"], inter, h, "mlp_in"), ("up", case["mlp"], inter, h, "mlp_in"),
            ("down", case["down"], h, inter, "mlp_mid")]


def prepare(case, seed):
    dev = torch.device("cuda")
    state = {"case": case, "x": {}, "w": {}}
    for i, (label, qtype, n, k, act) in enumerate(_weights(case)):
        state["w"][label] = (synth.make_weight_on_device(n, k, QT[qtype], 100 * seed + i, dev), act)
        if case["m"] and act not in state["x"]:
            g = torch.Generator(device=dev)
            g.manual_seed(100 * seed + 50 + i)
            state["x"][act] = torch.randn((case["m"], k), device=dev, generator=g).to(torch.bfloat16)
    if case["op"] == "train":
        g = torch.Generator(device=dev)
        g.manual_seed(100 * seed + 99)
        state["g"] = torch.randn((case["m"], case["n"]), device=dev, generator=g).to(torch.bfloat16)
        state["x"]["x"].requires_grad_(True)
    return state


def run(state):
    case = state["case"]
    if case["op"] == "dequantize":
        return state["w"]["w"][0].dequantize(getattr(torch, case["dtype"]))
    if case["op"] == "train":
        x, w = state["x"]["x"], state["w"]["w"][0]
        y = gj.matmul(x, w)
        (dx,) = torch.autograd.grad(y, x, state["g"])
        return [y.detach(), dx]
    xs = state["x"]
    return [gj.matmul(xs[act], w) for w, act in state["w"].values()]


def work(case):
    total, flops, seen = 0, 0, set()
    for _, qtype, n, k, act in _weights(case):
        bs, ts = _gguf.GGML_QUANT_SIZES[QT[qtype]]
        total += n * (k // bs) * ts
        if case["op"] == "dequantize":
            return {"bytes": total + n * k * (4 if case["dtype"] == "float32" else 2), "flops": n * k}
        m = case["m"]
        total += 2 * m * n + (0 if act in seen else 2 * m * k)
        seen.add(act)
        flops += 2 * m * n * k
    return {"bytes": 2 * total if case["op"] == "train" else total, "flops": 2 * flops if case["op"] == "train" else flops}


def tolerance(case):
    # Decoding is defined bit for bit (float32 arithmetic of the format, rounded once to the output type).
    if case["op"] == "dequantize":
        return "exact"
    # bf16 results of float32 sums over weights that are exact, or rounded once to bf16 as the package's dense route and
    # its tensor-core route do: 1.7e-3 and 2.4e-3 off the exact product, 2.9e-3 from one another in the 2-norm; the
    # largest single difference is one bf16 step of a value plus about five sigma of the weights' rounding.
    return {"rel": 8e-3, "max": 4e-2}


def _dense(w):
    """Float32 decode of a weight by gguf's numpy code, as float64 on the GPU, in row slabs on the host's cores."""
    data = w.data.cpu().numpy()
    n, k = w.shape
    if w.qtype.name.startswith("IQ"):
        _gguf.dequantize(data[:1], w.qtype)         # loads the format's grid once
    rows = max(1, (1 << 20) // k)
    out = torch.empty((n, k), dtype=torch.float64, device="cuda")

    def one(r):
        return r, np.asarray(_gguf.dequantize(data[r:r + rows], w.qtype), dtype=np.float32).reshape(-1, k)

    with concurrent.futures.ThreadPoolExecutor() as pool, np.errstate(all="ignore"):
        for r, part in pool.map(one, range(0, n, rows)):
            out[r:r + len(part)] = torch.from_numpy(part).cuda()
    return out


def exact(case, seed):
    state = prepare(case, seed)
    if case["op"] == "dequantize":
        return _dense(state["w"]["w"][0])
    if case["op"] == "train":
        dense = _dense(state["w"]["w"][0])
        return [state["x"]["x"].detach().double() @ dense.T, state["g"].double() @ dense]
    return [state["x"][act].double() @ _dense(w).T for w, act in state["w"].values()]
