"""The work a program has this framework do, as cases that can be timed: packed-weight products from one activation row to a
prefill batch, routed expert layers, greedy decoding of a dense model, and loading a packed tensor.

``listed()`` are fixed cases, ``draw(rng)`` gives others of the same ranges.  ``prepare`` builds what a program holds before
the call -- the loaded model, which does not depend on the seed, and the inputs, which do -- and ``run`` is one pass
through the public entry points."""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tyloquant_b200 import QuantWeight, decoder, encode, moe

DEV = "cuda:0"

# weight formats: (label of the record, bits, group size, sub-scale bits), or the lattice records
FORMATS = {
    "NINT2": (2, 16, 5), "NINT3": (3, 24, 5), "NINT4": (4, 24, 6), "NINT5": (5, 28, 7), "NINT6": (6, 24, 7), "NINT8": (8, 48, 7),
    "NINT4-32": (4, 32, 6), "NINT8-32": (8, 32, 7), "NVQ3": None, "NVQ3J-512": None,
}
STREAM_BYTES = 160e6   # a pass over weights of this size leaves nothing of them in the L2 cache for the next pass


def _linear(name, fmt, m, n, k, layers):
    return {"name": name, "kind": "linear", "fmt": fmt, "m": m, "n": n, "k": k, "layers": layers}


def _moe(name, tokens, experts, routes, hidden, ffn, widths):
    return {"name": name, "kind": "moe", "tokens": tokens, "experts": experts, "routes": routes, "hidden": hidden, "ffn": ffn, "widths": widths}


def _decode(name, batch, context, layers, hidden, kv_heads, ffn, vocab, attn, mlp):
    return {"name": name, "kind": "decode", "batch": batch, "context": context, "layers": layers, "hidden": hidden, "kv_heads": kv_heads,
            "ffn": ffn, "vocab": vocab, "attn": attn, "mlp": mlp}


def listed():
    return [
        # one row through one small matrix, called on its own: what a single product costs its caller
        _linear("row_nint3_4096", "NINT3", 1, 4096, 4096, 1),
        # a few sequences decoding together, lattice weights, the same projection of successive layers
        _linear("rows8_nvq3_17408x5120", "NVQ3", 8, 17408, 5120, 4),
        # the largest batch of the weight-streaming kernels, long rows (a down projection)
        _linear("rows16_nint6_4096x14336", "NINT6", 16, 4096, 14336, 4),
        # a short prompt: ragged in every dimension, a group size that is no multiple of eight
        _linear("prompt77_nint5_5000x2888", "NINT5", 77, 5000, 2888, 4),
        # prefill of 512 tokens, scalar codes
        _linear("prefill512_nint4_14336x4096", "NINT4-32", 512, 14336, 4096, 2),
        # prefill with lattice weights
        _linear("prefill256_nvq3j_17408x5120", "NVQ3J-512", 256, 17408, 5120, 1),
        # an expert layer with mixed code widths: one decoding sequence, a decoding batch, a prompt
        _moe("experts_1_token", 1, 128, 8, 2048, 768, "2346"),
        _moe("experts_32_tokens", 32, 128, 8, 2048, 768, "2346"),
        _moe("experts_256_tokens", 256, 128, 8, 2048, 768, "2346"),
        # greedy decoding of an 8B-shaped dense model at a 4096-token context, one sequence and sixteen
        _decode("decode_batch1", 1, 4096, 32, 4096, 8, 14336, 128256, "NINT4", "NINT6"),
        _decode("decode_batch16", 16, 4096, 32, 4096, 8, 14336, 128256, "NINT4", "NINT6"),
        # model loading: a packed record in host memory to the device and decoded
        {"name": "load_nint6_14336x4096", "kind": "load", "fmt": "NINT6", "n": 14336, "k": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above; half of them plain products."""
    kind = rng.choice(["linear"] * 6 + ["moe"] * 3 + ["decode"] * 2 + ["load"])
    if kind == "moe":
        return {"kind": "moe", "tokens": _log_int(rng, 1, 1024), "experts": rng.choice([32, 64, 128]), "routes": rng.choice([2, 4, 6, 8]),
                "hidden": 8 * _log_int(rng, 128, 320), "ffn": 8 * _log_int(rng, 48, 128), "widths": rng.choice(["2346", "2346", "46", "3458"])}
    if kind == "decode":
        hidden, kv_heads = rng.choice([(4096, 8), (4096, 8), (2048, 4)])
        return {"kind": "decode", "batch": _log_int(rng, 1, 16), "context": _log_int(rng, 100, 4096), "layers": _log_int(rng, 4, 32), "hidden": hidden,
                "kv_heads": kv_heads, "ffn": 16 * _log_int(rng, 256, 896), "vocab": _log_int(rng, 16000, 128256),
                "attn": rng.choice(["NINT4", "NINT3", "NINT6"]), "mlp": rng.choice(["NINT6", "NINT4", "NINT3"])}
    fmt = rng.choice(sorted(FORMATS))
    n, k = _log_int(rng, 512, 17408), _log_int(rng, 512, 14336)
    if rng.random() < 0.8:
        k = (k + 7) // 8 * 8
    if n * k > 90e6:
        n = int(90e6 / k)
    if kind == "load":
        return {"kind": "load", "fmt": fmt, "n": n, "k": k}
    layers = 1 if rng.random() < 0.4 else max(1, min(8, int(STREAM_BYTES / _payload(fmt, n, k))))
    return {"kind": "linear", "fmt": fmt, "m": _log_int(rng, 1, 2048), "n": n, "k": k, "layers": layers}


# ---- the model: packed records of seeded N(0, 0.02) weights, as the benchmark makes them -----------------------------------

def _bits(count):
    return (int(count) + 7) // 8


def _payload(fmt, n, k):
    """Bytes of a record's file streams."""
    if FORMATS[fmt] is None:
        ng = -(-k // 24)
        index_bits, tables = (8, 0) if fmt == "NVQ3" else (9, 64 + 2 * 512 * 4)
        return 2 * n + _bits(4 * n * ng) + _bits(index_bits * n * -(-k // 4)) + _bits(7 * n * -(-k // 8)) + tables
    bits, gs, sub = FORMATS[fmt]
    ng = -(-k // gs)
    return 4 * n + 2 * _bits(sub * n * ng) + _bits(bits * n * ng * gs)


def _randn(shape, seed, scale=1.0):
    gen = torch.Generator(DEV).manual_seed(seed)
    return torch.randn(shape, device=DEV, generator=gen) * scale


def _blob(fmt, n, k, seed):
    w = _randn((n, k), seed, 0.02).to(torch.bfloat16).float()
    if FORMATS[fmt] is None:
        jsc = fmt != "NVQ3"
        banks = encode.synthetic_d4_banks(512, 2, seed=9) if jsc else encode.d4_256_codebook()[None]
        return encode.nvq_blob(encode.quantize_nvq3(w.cpu().numpy(), banks, jsc=jsc, device=DEV))
    bits, gs, sub = FORMATS[fmt]
    return encode.nint_blob(encode.quantize_nint(w, bits, gs, sub, device=DEV))


def _label(fmt):
    return fmt.partition("-")[0] if fmt.startswith("NINT") else fmt


@functools.lru_cache(maxsize=3)
def _linear_weights(fmt, n, k, layers):
    blob = _blob(fmt, n, k, 1001)
    return [QuantWeight.from_blob(_label(fmt), blob) for _ in range(layers)]   # every layer streams memory of its own


@functools.lru_cache(maxsize=1)
def _experts(experts, hidden, ffn, widths):
    bits = np.random.default_rng(4003).choice([int(c) for c in widths], experts)
    pair = []
    for seed, shape in ((4001, (experts, 2 * ffn, hidden)), (4002, (experts, hidden, ffn))):
        pair.append(moe.MoeWeight(encode.quantize_expertwise(_randn(shape, seed, 0.02).to(torch.bfloat16).float(), bits, device=DEV)))
    return bits, pair[0], pair[1]


STEPS = 8   # tokens decoded per pass


@functools.lru_cache(maxsize=1)
def _model(layers, hidden, kv_heads, ffn, vocab, attn, mlp, context, batch):
    heads = hidden // 128
    dec = decoder.Decoder(hidden=hidden, n_q_heads=heads, n_kv_heads=kv_heads, ffn=ffn, vocab=vocab, layers=layers,
                          max_ctx=context + STEPS + 8, max_batch=batch)
    shapes = (((heads + 2 * kv_heads) * 128, hidden, attn), (hidden, hidden, attn), (2 * ffn, hidden, mlp), (hidden, ffn, mlp))
    first = [QuantWeight.from_blob(_label(f), _blob(f, n, k, 5000 + i)) for i, (n, k, f) in enumerate(shapes)]
    dec.set_layer(0, *first)
    for i in range(1, layers):   # the other blocks are device copies: each streams memory of its own
        dec.set_layer(i, *[w.clone() for w in first])
    dec.set_head(QuantWeight.from_blob(_label(mlp), _blob(mlp, vocab, hidden, 5009)), _randn((vocab, hidden), 5010).to(torch.bfloat16))
    return dec


# ---- the interface ---------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "linear":
        return {"kind": "linear", "weights": _linear_weights(case["fmt"], case["n"], case["k"], case["layers"]),
                "xs": [_randn((case["m"], case["k"]), 7919 * seed + i).to(torch.bfloat16) for i in range(case["layers"])]}
    if case["kind"] == "moe":
        _, gate_up, down = _experts(case["experts"], case["hidden"], case["ffn"], case["widths"])
        return {"kind": "moe", "gate_up": gate_up, "down": down, "routes": case["routes"],
                "x": _randn((case["tokens"], case["hidden"]), seed).to(torch.bfloat16), "logits": _randn((case["tokens"], case["experts"]), seed + 1)}
    if case["kind"] == "decode":
        dec = _model(case["layers"], case["hidden"], case["kv_heads"], case["ffn"], case["vocab"], case["attn"], case["mlp"], case["context"],
                     case["batch"])
        ids = torch.randint(0, case["vocab"], (STEPS, case["batch"]), device=DEV, generator=torch.Generator(DEV).manual_seed(seed), dtype=torch.int32)
        return {"kind": "decode", "dec": dec, "context": case["context"], "batch": case["batch"], "fill": seed & 0x7FFFFFFF, "ids": list(ids)}
    return {"kind": "load", "label": _label(case["fmt"]), "blob": _blob(case["fmt"], case["n"], case["k"], seed)}


def run(state):
    if state["kind"] == "linear":
        return [w.matmul(x) for w, x in zip(state["weights"], state["xs"])]
    if state["kind"] == "moe":
        ids, weights = moe.moe_topk(state["logits"], state["routes"])
        y = moe.moe_ffn(state["gate_up"], state["down"], state["x"], ids, weights, out_dtype=torch.bfloat16)
        return {"ids": ids, "weights": weights, "y": y}
    if state["kind"] == "decode":
        # the cache fill stands in for the prompt's prefill and sets the positions; the tokens are given, so that the logits
        # of a step do not hang on a near tie of the step before
        dec, logits = state["dec"], []
        dec.fill_cache(state["context"], state["fill"])
        for ids in state["ids"]:
            dec.step(ids)
            logits.append(dec.read_logits(state["batch"]))
        return logits
    w = QuantWeight.from_blob(state["label"], state["blob"])
    return w.dequantize()


def work(case):
    if case["kind"] == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": case["layers"] * (_payload(case["fmt"], n, k) + 2 * m * (n + k)), "flops": case["layers"] * 2.0 * m * n * k}
    if case["kind"] == "moe":
        t, e, r, h, f = case["tokens"], case["experts"], case["routes"], case["hidden"], case["ffn"]
        bits = np.random.default_rng(4003).choice([int(c) for c in case["widths"]], e)
        every = sum(_payload("NINT%d" % b, 2 * f, h) + _payload("NINT%d" % b, h, f) for b in bits)
        touched = 1.0 - (1.0 - r / e) ** t   # share of the experts that t tokens are expected to use
        return {"bytes": every * touched + 4 * t * (h + e + 2 * r), "flops": 6.0 * t * r * h * f}
    if case["kind"] == "decode":
        h, f, d, b = case["hidden"], case["ffn"], case["kv_heads"] * 128, case["batch"]
        weights = case["layers"] * (_payload(case["attn"], h + 2 * d, h) + _payload(case["attn"], h, h) + _payload(case["mlp"], 2 * f, h) +
                                    _payload(case["mlp"], h, f)) + _payload(case["mlp"], case["vocab"], h)
        params = case["layers"] * ((h + 2 * d) * h + h * h + 3 * f * h) + case["vocab"] * h
        cache = 4 * case["layers"] * d * case["context"] * b
        attention = 4.0 * case["layers"] * h * case["context"] * b
        return {"bytes": STEPS * (weights + cache + 8 * b * case["vocab"]) + cache, "flops": STEPS * (2.0 * params * b + attention)}
    return {"bytes": _payload(case["fmt"], case["n"], case["k"]) + 4 * case["n"] * case["k"], "flops": 0.0}


def tolerance(case):
    if case["kind"] == "load":
        return "exact"          # the decoder is bit-identical to the format's definition
    if case["kind"] == "decode":
        return {"rel": 2e-2}    # bf16 activations between the products of every block: one rounding more or less spreads over 32 blocks
    return {"rel": 4e-3}        # bf16 outputs; expert ids are whole numbers and stay exact
