"""Workloads of the library, through its public Python entry points, for timing one build against another.

    listed()                the cases that are looked at one by one
    draw(rng)               another case of the same ranges
    prepare(case, seed)     what a program holds before the call: packed layers, activations, caches, a captured step
    run(state)              one pass
    work(case)              bytes and floating-point operations that a pass cannot do without
    tolerance(case)         how far another correct implementation of the same precision may be off

Five kinds of work:

    linear    one quantized linear, `QLinear.forward`: y[M, N] = x[M, K] . dequant(W)^T
    block     the four linears of one decoder layer in turn (QKV, O, gate+up, down with its SiLU * up), called one
              by one as a serving stack without graphs does
    decode    one token per sequence through a few layers of the decoder and the output projection, replayed from
              a CUDA graph or called eagerly
    prefill   the prompt of each sequence through the same decoder
    convert   a GPTQ checkpoint tensor or an fp16 weight into a packed layer, as at model load

Imported with the repository root as the working folder.
"""
from __future__ import annotations

import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "qfactory-ae_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from qfactory import QLinear  # noqa: E402
from qfactory.decoder import DecoderConfig, QuantDecoder  # noqa: E402
from qfactory.gptq import layer_from_gptq  # noqa: E402

# Llama-2-70B widths; a case takes as many of its 80 identical layers as it says
D_MODEL, HEADS, KV_HEADS, D_FF, VOCAB, MAX_LEN = 8192, 64, 8, 28672, 32000, 512


def listed():
    return [
        # one token through the smallest layer of a 7B model: launch latency and host time
        {"name": "linear_o_m1", "kind": "linear", "m": 1, "n": 4096, "k": 4096, "bits": 4, "group": 128, "sym": False},
        # interactive decode of a 7B model, one sequence: the linears of a layer
        {"name": "block_7b_m1", "kind": "block", "m": 1, "d": 4096, "ff": 11008, "bits": 4, "group": 128},
        # the same with a batch of sixteen sequences
        {"name": "block_7b_m16", "kind": "block", "m": 16, "d": 4096, "ff": 11008, "bits": 4, "group": 128},
        # 3-bit weights, a few sequences
        {"name": "linear_b3_m4", "kind": "linear", "m": 4, "n": 8192, "k": 8192, "bits": 3, "group": 128, "sym": False},
        # 8-bit symmetric weights, a batch between decode and prefill sizes
        {"name": "linear_b8_m24", "kind": "linear", "m": 24, "n": 8192, "k": 8192, "bits": 8, "group": 128, "sym": True},
        # a shard of a row-parallel layer whose K (11008 / 4) is an odd multiple of 64, N no multiple of the tile,
        # a short prompt of odd length
        {"name": "linear_ragged_m37", "kind": "linear", "m": 37, "n": 3000, "k": 2752, "bits": 4, "group": 64, "sym": False},
        # 70B MLP layers at a large decode batch, a short prompt and a long one
        {"name": "linear_up_m64", "kind": "linear", "m": 64, "n": 28672, "k": 8192, "bits": 4, "group": 128, "sym": False},
        {"name": "linear_down_m128", "kind": "linear", "m": 128, "n": 8192, "k": 28672, "bits": 4, "group": 128, "sym": False},
        {"name": "linear_up_m1024", "kind": "linear", "m": 1024, "n": 28672, "k": 8192, "bits": 4, "group": 128, "sym": False},
        # one decode step of one sequence, a tenth of the 70B decoder, from a CUDA graph
        {"name": "decode_b1", "kind": "decode", "batch": 1, "layers": 8, "pos": 255, "graph": True},
        # the prompt of 128 tokens in front of it
        {"name": "prefill_128", "kind": "prefill", "batch": 1, "layers": 8, "tokens": 128},
        # model load: a GPTQ checkpoint's down projection into a packed layer
        {"name": "convert_gptq", "kind": "convert", "source": "gptq", "n": 8192, "k": 28672, "bits": 4, "group": 128, "sym": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _bits_group_sym(rng):
    bits = rng.choice((4, 4, 4, 4, 2, 3, 8))
    group = rng.choice((128, 128, 128, 64, 256, -1))
    return bits, 128 if bits == 3 and group == 64 else group, rng.random() < 0.3


def draw(rng):
    kind = rng.choices(("linear", "block", "decode", "prefill", "convert"), (12, 3, 2, 1, 2))[0]
    if kind == "linear":
        bits, group, sym = _bits_group_sym(rng)
        n = _log_int(rng, 1024, 32768)
        if rng.random() < 0.75:
            n = max(1024, n // 128 * 128)
        # K in whole groups; 64-code groups give the odd multiples of 64 too
        unit = 64 if group == 64 else 128 if group == -1 else group
        k = max(1024, _log_int(rng, 1024, 32768) // unit * unit)
        m = rng.choice((1, 1, _log_int(rng, 2, 16), _log_int(rng, 2, 16), _log_int(rng, 17, 1024), _log_int(rng, 17, 1024)))
        m = max(1, min(m, 1024 * 28672 * 8192 // (n * k)))
        if k % 128:
            m = min(m, 256)
        return {"kind": kind, "m": m, "n": n, "k": k, "bits": bits, "group": group, "sym": sym}
    if kind == "block":
        d = 256 * rng.randint(8, 32)
        return {"kind": kind, "m": rng.choice((1, _log_int(rng, 1, 64), _log_int(rng, 1, 256))), "d": d,
                "ff": max(256, int(d * rng.uniform(2.5, 3.7)) // 256 * 256),
                "bits": rng.choice((4, 4, 4, 2, 3, 8)), "group": rng.choice((128, 128, 256))}
    layers = rng.randint(2, 8)
    if kind == "decode":
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "layers": layers, "pos": rng.randint(1, MAX_LEN - 1),
                "graph": rng.random() < 0.7}
    if kind == "prefill":
        batch = rng.choice((1, 1, 2, 4))
        return {"kind": kind, "batch": batch, "layers": min(layers, 6), "tokens": rng.randint(16, 128 // batch)}
    bits, group, sym = _bits_group_sym(rng)
    source = "gptq" if bits != 3 and rng.random() < 0.6 else "float"
    unit = group if group > 0 else 128
    return {"kind": kind, "source": source, "n": _log_int(rng, 1024, 8192) // 32 * 32,
            "k": max(1024, _log_int(rng, 1024, 28672) // unit * unit), "bits": bits, "group": unit,
            "sym": sym and source == "gptq"}


# ---- inputs --------------------------------------------------------------------------------------

def _layer(m, n, k, bits, group, sym, gen):
    """Codes and zero points uniform, scales U(0.002, 0.02): a packed layer made for m rows."""
    codes = torch.randint(0, 1 << bits, (k, n), generator=gen, dtype=torch.int32, device="cuda")
    if group == -1:
        return QLinear.init(m, k, n, bits, codes)
    scales = (torch.rand(k // group, n, generator=gen, device="cuda") * 0.018 + 0.002).half()
    zeros = None if sym else torch.randint(0, 1 << bits, (k // group, n), generator=gen, dtype=torch.int32, device="cuda")
    return QLinear.init(m, k, n, bits, codes, group, scales, zeros)


def _acts(m, k, gen, scale=1.0):
    return (torch.randn(m, k, generator=gen, device="cuda") * scale).half()


def _block_shapes(case):
    d, ff = case["d"], case["ff"]
    return [(3 * d, d), (d, d), (2 * ff, d), (d, ff)]


def _words(case, gen, shape):
    """Random int32 words: every packed field of a GPTQ tensor uniform."""
    return torch.randint(-2 ** 31, 2 ** 31, shape, generator=gen, dtype=torch.int64, device="cuda").to(torch.int32)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "linear":
        # raw codes (no scales) are tens of times larger than scaled weights: the activations keep y in fp16's range
        scale = 1.0 if case["group"] != -1 else 2.0 ** -case["bits"]
        return {"kind": kind, "x": _acts(case["m"], case["k"], gen, scale),
                "layer": _layer(case["m"], case["n"], case["k"], case["bits"], case["group"], case["sym"], gen)}
    if kind == "block":
        m, d = case["m"], case["d"]
        layers = [_layer(m, n, k, case["bits"], case["group"], False, gen) for n, k in _block_shapes(case)]
        if case["bits"] == 8:   # 8-bit codes carry sixteen times finer scales than 4-bit ones
            for layer in layers:
                layer.s.mul_(1.0 / 16)
        return {"kind": kind, "layers": layers, "x": _acts(m, d, gen), "att": _acts(m, d, gen), "h": _acts(m, d, gen)}
    if kind in ("decode", "prefill"):
        cfg = DecoderConfig(layers=case["layers"], d_model=D_MODEL, n_heads=HEADS, n_kv_heads=KV_HEADS, d_ff=D_FF,
                            vocab=VOCAB, max_len=MAX_LEN)
        model = QuantDecoder(cfg, seed=seed, batch=case["batch"])
        state = {"kind": kind, "model": model, "graph": None}
        tokens = 1 if kind == "decode" else case["tokens"]
        state["tokens"] = torch.randint(0, VOCAB, (case["batch"], tokens), generator=gen, device="cuda")
        if kind == "prefill":
            state["pos"] = torch.arange(tokens, device="cuda")
            return state
        # the keys and values of the tokens before this one
        for cache in (model.k_cache, model.v_cache):
            cache[..., : case["pos"], :].normal_(generator=gen)
        state["pos"] = torch.full((1,), case["pos"], dtype=torch.long, device="cuda")
        if case["graph"]:
            with torch.no_grad():
                side = torch.cuda.Stream()
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    model(state["tokens"], state["pos"])
                torch.cuda.current_stream().wait_stream(side)
                state["graph"] = torch.cuda.CUDAGraph()
                with torch.cuda.graph(state["graph"]):
                    state["logits"] = model(state["tokens"], state["pos"])
        return state
    n, k, bits, group = case["n"], case["k"], case["bits"], case["group"]
    if case["source"] == "float":
        return {"kind": kind, "source": "float", "weight": _acts(k, n, gen, k ** -0.5), "bits": bits, "group": group}
    pf = 32 // bits
    return {"kind": kind, "source": "gptq", "bits": bits, "group": group, "sym": case["sym"],
            "qweight": _words(case, gen, (k // pf, n)), "qzeros": _words(case, gen, (k // group, n // pf)),
            "scales": (torch.rand(k // group, n, generator=gen, device="cuda") * 0.018 + 0.002).half()}


# ---- one pass ------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["layer"](state["x"])
    if kind == "block":
        qkv, o, gate_up, down = state["layers"]
        a, b, gu = qkv(state["x"]), o(state["att"]), gate_up(state["h"])
        return [a, b, gu, down.forward_silu_mul(gu)]
    if kind in ("decode", "prefill"):
        model = state["model"]
        if state["graph"] is not None:
            state["graph"].replay()
            logits = state["logits"]
        else:
            logits = model(state["tokens"], state["pos"])
        return {"logits": logits, "k_cache": model.k_cache, "v_cache": model.v_cache}
    if state["source"] == "float":
        layer = QLinear.from_float(state["weight"], state["bits"], state["group"])
    else:
        layer = layer_from_gptq(state["qweight"], state["qzeros"], state["scales"], state["bits"], state["group"],
                                sym=state["sym"])
    return {"w": layer.w, "s": layer.s, "z": layer.z}


# ---- what a pass cannot do without ---------------------------------------------------------------

def _weight_bytes(n, k, bits, group, sym=False):
    groups = 0 if group == -1 else k // group
    return n * k * bits / 8 + groups * n * 2 + (0 if sym else groups * n * bits / 8)


def _linear_work(m, n, k, bits, group, sym=False):
    return _weight_bytes(n, k, bits, group, sym) + 2 * m * (n + k), 2 * m * n * k


def work(case):
    kind = case["kind"]
    if kind == "linear":
        nbytes, flops = _linear_work(case["m"], case["n"], case["k"], case["bits"], case["group"], case["sym"])
        return {"bytes": nbytes, "flops": flops}
    if kind == "block":
        parts = [_linear_work(case["m"], n, k, case["bits"], case["group"]) for n, k in _block_shapes(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind in ("decode", "prefill"):
        b, t = case["batch"], 1 if kind == "decode" else case["tokens"]
        past = case["pos"] if kind == "decode" else 0
        hd = D_MODEL // HEADS
        shapes = [(D_MODEL + 2 * KV_HEADS * hd, D_MODEL), (D_MODEL, D_MODEL), (2 * D_FF, D_MODEL), (D_MODEL, D_FF)]
        # weights once, cached keys and values read, new ones written; each token attends to itself and all before it
        nbytes = sum(_weight_bytes(n, k, 4, 128) for n, k in shapes) + 2 * b * KV_HEADS * hd * 2 * (past + t)
        flops = sum(2 * b * t * n * k for n, k in shapes) + 4 * b * HEADS * hd * (t * past + t * (t + 1) // 2)
        head = _linear_work(b, VOCAB, D_MODEL, 4, 128)
        return {"bytes": case["layers"] * nbytes + head[0] + 2 * b * t * D_MODEL, "flops": case["layers"] * flops + head[1]}
    packed = _weight_bytes(case["n"], case["k"], case["bits"], case["group"], case["sym"])
    source = 2 * case["n"] * case["k"] if case["source"] == "float" else packed
    return {"bytes": source + packed, "flops": 0}


def tolerance(case):
    if case["kind"] == "convert":
        return "exact"
    # fp16 operands and results, fp32 sums: 2^-11 for each rounding of a result, a dequantised weight or an
    # activation, and the same again where a result feeds the next product; the decoder chains several layers
    if case["kind"] == "linear":
        return {"rel": 1e-3}
    if case["kind"] == "block":
        return {"rel": 2e-3}
    return {"rel": 5e-3}
