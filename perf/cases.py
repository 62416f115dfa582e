"""The work that programs give this library, as cases that can be timed and whose results can be compared.

Seven kinds of pass, each through the package's public calls and, for the decoder glue, the C functions of
include/turboquant_c/turboquant_b200.h:

  linear    one or several TQ8 layers on an activation each: single projections, an LM head, host callers
  project   the seven projections of a decoder layer with RMSNorm, rotary embedding, SwiGLU and the residual sums:
            decode batches, prompt chunks, whole prompts
  step      a decoder layer's decode step: the same plus the KV append and attention over the compressed cache
  attend    KV append and attention of one layer for a batch of long sequences
  window    the fp16 decode window: one token slid in, hybrid attention over the window
  prompt    a new sequence's KV cache: created, filled with the prompt's keys and values, attended once and
            decompressed (what fills the fp16 window), released
  convert   a weight matrix through the converter's steps: codebook fit, quantisation, layer, fp16 weights back

Shapes are those of bench.py (4096 x 4096 layers, Qwen2.5-7B- and 32B-shaped decoder layers, the 151936 x 2048 LM
head, 3.5-bit caches of 4 or 8 KV heads at 4k to 128k tokens) and of the tests; draw() spreads over the same ranges.
"""
import ctypes as C
import math

import torch

import turboquant_mlx_core_b200 as tq

DEV = "cuda"
EPS, THETA = 1e-6, 1e6
ROOM = 16384                   # tokens of room that a decode loop keeps ahead of each sequence


def _layer_shape(hidden, inter, q_heads, kv_heads):
    return {"hidden": hidden, "inter": inter, "q_heads": q_heads, "kv_heads": kv_heads, "dim": 128}


LAYER_7B = _layer_shape(3584, 18944, 28, 4)
LAYER_32B = _layer_shape(5120, 27648, 40, 8)


def listed():
    return [
        # the smallest call: one projection for one token, fp32 activation and result in host memory, as a
        # binding without device buffers calls it
        {"name": "linear_host_b1", "kind": "linear", "in": 4096, "out": 4096, "layers": 1, "rows": 1, "block": 128,
         "shared": True, "host": True},
        # one projection of each of eight layers for one token: the headline shape, weights from HBM
        {"name": "linear_b1", "kind": "linear", "in": 4096, "out": 4096, "layers": 8, "rows": 1, "block": 128,
         "shared": True, "host": False},
        # checkpoints with two rotations (the quantiser's default configuration), a few sequences
        {"name": "linear_dual_b4", "kind": "linear", "in": 3584, "out": 3584, "layers": 8, "rows": 4, "block": 512,
         "shared": False, "host": False},
        # LM head for a small decode batch
        {"name": "lm_head_b8", "kind": "linear", "in": 2048, "out": 151936, "layers": 1, "rows": 8, "block": 128,
         "shared": True, "host": False},
        # a decode step of one user
        {"name": "step_7b_b1", "kind": "step", **LAYER_7B, "rows": 1, "context": 4096},
        # a decode step of a served batch on the larger model
        {"name": "step_32b_b32", "kind": "step", **LAYER_32B, "rows": 32, "context": 8192},
        # a large decode batch, or a short prompt chunk
        {"name": "project_7b_64", "kind": "project", **LAYER_7B, "rows": 64},
        # a prompt
        {"name": "project_7b_2048", "kind": "project", **LAYER_7B, "rows": 2048},
        # long-context decode attention of a batch
        {"name": "attend_16x32k", "kind": "attend", "seqs": 16, "context": 32768, "q_heads": 28, "kv_heads": 4,
         "dim": 128, "qjl": True},
        # the decode window at its default size
        {"name": "window_128k", "kind": "window", "context": 131072, "q_heads": 28, "kv_heads": 4, "dim": 128},
        # a new sequence with a long prompt, four layers of it
        {"name": "prompt_8k", "kind": "prompt", "tokens": 8192, "layers": 4, "q_heads": 28, "kv_heads": 4, "dim": 128,
         "f16": True},
        # the converter on one projection
        {"name": "convert_4096", "kind": "convert", "in": 4096, "out": 4096, "block": 512, "shared": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, lo, hi, step):
    return max(lo, min(hi, _log_int(rng, lo, hi) // step * step))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "project", "project", "step", "step", "attend", "attend", "window",
                       "prompt", "convert"])
    if kind == "linear":
        while True:
            n_in = _multiple(rng, 1024, 28672, 64)
            n_out = _log_int(rng, 512, 152064)
            host = rng.random() < 0.2
            rows = _log_int(rng, 1, 8 if host else 2048)
            if n_in * n_out <= 320e6 and rows * n_in * n_out <= 0.12e12:
                break
        shared = rng.random() < 0.75
        # enough layers that their weights do not stay in the L2 cache between passes, as in a model
        layers = 1 if host else max(1, min(16, int(64e6 / (n_in * n_out))))
        return {"kind": kind, "in": n_in, "out": n_out, "layers": layers, "rows": rows,
                "block": tq.adaptive_block_size(n_in, rng.choice([128, 512])), "shared": shared, "host": host}
    if kind in ("project", "step"):
        dim = 128
        kv_heads = rng.choice([2, 4, 8])
        q_heads = kv_heads * rng.choice([1, 4, 5, 7, 8])
        hidden = max(1024, min(5120, q_heads * dim))
        inter = _multiple(rng, 2 * hidden, min(6 * hidden, 27648), 64)
        shape = {"hidden": hidden, "inter": inter, "q_heads": q_heads, "kv_heads": kv_heads, "dim": dim}
        if kind == "project":
            return {"kind": kind, **shape, "rows": _log_int(rng, 2, 1024)}
        return {"kind": kind, **shape, "rows": _log_int(rng, 1, 32), "context": _log_int(rng, 128, 8192)}
    if kind == "attend":
        kv_heads = rng.choice([1, 2, 4, 8])
        q_heads = kv_heads * rng.choice([1, 4, 5, 7, 8])
        context = _log_int(rng, 256, 131072)
        seqs = _log_int(rng, 1, max(1, min(64, int(16 * 32768 * 4 / (context * kv_heads)))))
        return {"kind": kind, "seqs": seqs, "context": context, "q_heads": q_heads, "kv_heads": kv_heads,
                "dim": rng.choice([128, 128, 128, 64]), "qjl": rng.random() < 0.75}
    if kind == "window":
        kv_heads = rng.choice([1, 2, 4, 8])
        return {"kind": kind, "context": _log_int(rng, 256, 131072 * 4 // max(kv_heads, 4)),
                "q_heads": kv_heads * rng.choice([1, 4, 5, 7, 8]), "kv_heads": kv_heads, "dim": rng.choice([128, 128, 128, 64])}
    if kind == "prompt":
        kv_heads = rng.choice([2, 4, 8])
        return {"kind": kind, "tokens": _log_int(rng, 16, 8192 * 4 // max(kv_heads, 4)), "layers": rng.choice([1, 2, 4]),
                "q_heads": kv_heads * rng.choice([1, 4, 7]), "kv_heads": kv_heads, "dim": rng.choice([128, 128, 128, 64]),
                "f16": rng.random() < 0.75}
    n_in = _multiple(rng, 512, 8192, 64)
    n_out = _log_int(rng, 256, min(8192, 16777216 // n_in))
    return {"kind": kind, "in": n_in, "out": n_out, "block": tq.adaptive_block_size(n_in, rng.choice([128, 512])),
            "shared": rng.random() < 0.75}


# ---- inputs ----------------------------------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, shape, scale=1.0, dtype=torch.float16):
    return (torch.randn(shape, generator=g, device=DEV, dtype=torch.float32) * scale).to(dtype)


def _codebooks(g, block):
    """A layer's codebooks as the converter fits them, from a sample of its weights."""
    return tq.fit_layer_codebooks(_normal(g, (256, 4096), 0.02).float(), block, 4, 4, 100)


def _linear(g, n_in, n_out, block, shared, books):
    w = _normal(g, (n_out, n_in), 0.02).float()
    qw = tq.quantize_weight(w, books[0], books[1], tq.QuantizerConfig(4, 4, block, shared))
    return tq.TurboQuantLinear(n_in, n_out, qw, books[0], books[1], block)


def _kv(g, tokens, heads, dim, dtype=torch.float16):
    """Keys or values: N(0, 1) with 5 % of the channels scaled by 8."""
    wide = torch.randperm(dim, generator=g, device=DEV)[: max(1, dim // 20)]
    x = torch.randn((tokens, heads, dim), generator=g, device=DEV)
    x[..., wide] *= 8.0
    return x.to(dtype)


def _caches(g, case, seqs):
    caches = []
    for _ in range(seqs):
        c = tq.TQKVCache(1, case["kv_heads"], case["dim"])
        c.reserve(0, case["context"] + ROOM)
        c.append(0, _kv(g, case["context"], case["kv_heads"], case["dim"]), _kv(g, case["context"], case["kv_heads"], case["dim"]))
        caches.append(c)
    return caches


def _decoder_layer(g, case):
    hidden, inter, dim = case["hidden"], case["inter"], case["dim"]
    q_out, kv_out = case["q_heads"] * dim, case["kv_heads"] * dim

    def lin(n_in, n_out):
        block = tq.adaptive_block_size(n_in, 128)
        return _linear(g, n_in, n_out, block, True, books[block])

    books = {b: _codebooks(g, b) for b in {tq.adaptive_block_size(n, 128) for n in (hidden, q_out, inter)}}
    return {"q": lin(hidden, q_out), "k": lin(hidden, kv_out), "v": lin(hidden, kv_out), "o": lin(q_out, hidden),
            "gate_up": lin(hidden, 2 * inter), "down": lin(inter, hidden),
            "norm1": _normal(g, (hidden,), 0.1) + 1, "norm2": _normal(g, (hidden,), 0.1) + 1}


def prepare(case, seed):
    tq.load()
    g = _generator(seed)
    kind, state = case["kind"], {"case": case}
    if kind == "linear":
        books = _codebooks(g, case["block"])
        state["layers"] = [_linear(g, case["in"], case["out"], case["block"], case["shared"], books) for _ in range(case["layers"])]
        if case["host"]:
            state["x"] = [_normal(g, (case["rows"], case["in"]), dtype=torch.float32).cpu().numpy() for _ in state["layers"]]
        else:
            state["x"] = [_normal(g, (case["rows"], case["in"])) for _ in state["layers"]]
    elif kind in ("project", "step"):
        rows = case["rows"]
        state["w"] = _decoder_layer(g, case)
        state["x"] = _normal(g, (rows, case["hidden"]))
        if kind == "step":
            state["positions"] = torch.full((rows,), case["context"], device=DEV, dtype=torch.int32)
            state["caches"] = _caches(g, case, rows)
        else:
            state["positions"] = torch.arange(rows, device=DEV, dtype=torch.int32)
            state["attended"] = _normal(g, (rows, case["q_heads"] * case["dim"]), 0.1)
    elif kind == "attend":
        state["caches"] = _caches(g, case, case["seqs"])
        state["q"] = _normal(g, (case["seqs"], case["q_heads"], case["dim"]))
        state["k"] = _kv(g, case["seqs"], case["kv_heads"], case["dim"])
        state["v"] = _kv(g, case["seqs"], case["kv_heads"], case["dim"])
    elif kind == "window":
        n, heads, dim = case["context"], case["kv_heads"], case["dim"]
        k, v = _kv(g, n, heads, dim), _kv(g, n, heads, dim)
        state["cache"] = tq.TQKVCache(1, heads, dim)
        state["cache"].append(0, k, v)
        state["window"] = tq.DecodeBuffer(n, heads, dim)
        state["window"].rebuild(k, v)
        state["q"] = _normal(g, (case["q_heads"], dim))
        state["k"], state["v"] = _kv(g, 1, heads, dim), _kv(g, 1, heads, dim)
    elif kind == "prompt":
        n, heads, dim = case["tokens"], case["kv_heads"], case["dim"]
        dtype = torch.float16 if case["f16"] else torch.float32
        state["k"] = [_kv(g, n, heads, dim, dtype) for _ in range(case["layers"])]
        state["v"] = [_kv(g, n, heads, dim, dtype) for _ in range(case["layers"])]
        state["q"] = [_normal(g, (1, case["q_heads"], dim)) for _ in range(case["layers"])]
    else:
        state["w"] = _normal(g, (case["out"], case["in"]), 0.02).float()
    return state


# ---- one pass --------------------------------------------------------------------------------------------


def _p(t):
    return C.c_void_p(t.data_ptr())


def _first_norm_and_qkv(L, case, w, x, positions):
    rows = x.shape[0]
    n1 = torch.empty_like(x)
    tq._lib.check(L.tq_rmsnorm_f16(_p(x), _p(w["norm1"]), _p(n1), rows, case["hidden"], EPS, None), "rmsnorm")
    q, k, v = tq.forward_group([w["q"], w["k"], w["v"]], n1)
    tq._lib.check(L.tq_rope_qk_f16(_p(q), _p(k), _p(positions), rows, case["q_heads"], case["kv_heads"], case["dim"], THETA, None), "rope")
    return q, k, v


def _rest_of_layer(L, case, w, x, attended):
    rows, hidden = x.shape[0], case["hidden"]
    o = w["o"].forward(attended)
    h, n2 = torch.empty_like(x), torch.empty_like(x)
    tq._lib.check(L.tq_exchange_sum_f16_rmsnorm(_p(o), 1, rows * hidden, rows, hidden, _p(x), _p(h), _p(w["norm2"]), _p(n2), EPS, None), "sum")
    gate_up = w["gate_up"].forward(n2)
    act = torch.empty((rows, case["inter"]), device=DEV, dtype=torch.float16)
    tq._lib.check(L.tq_swiglu_f16(_p(gate_up), _p(act), rows, case["inter"], None), "swiglu")
    d = w["down"].forward(act)
    y = torch.empty_like(x)
    tq._lib.check(L.tq_exchange_sum_f16(_p(d), 1, rows * hidden, rows * hidden, _p(h), _p(y), None), "sum")
    return y


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        return [lin.forward(x) for lin, x in zip(state["layers"], state["x"])]
    if kind == "project":
        L = tq.load()
        q, k, v = _first_norm_and_qkv(L, case, state["w"], state["x"], state["positions"])
        return {"q": q, "k": k, "v": v, "hidden": _rest_of_layer(L, case, state["w"], state["x"], state["attended"])}
    if kind == "step":
        L = tq.load()
        rows, dim, caches = case["rows"], case["dim"], state["caches"]
        q, k, v = _first_norm_and_qkv(L, case, state["w"], state["x"], state["positions"])
        tq.append_batch(caches, 0, k.view(rows, case["kv_heads"], dim), v.view(rows, case["kv_heads"], dim))
        # the newest `context` tokens: every pass sees as many, although the sequences grow
        first = caches[0].seq_length() - case["context"]
        a = tq.compressed_attention(caches, 0, q.view(rows, case["q_heads"], dim), start=first, use_qjl=True)
        return {"k": k, "v": v, "attended": a,
                "hidden": _rest_of_layer(L, case, state["w"], state["x"], a.view(rows, case["q_heads"] * dim))}
    if kind == "attend":
        caches = state["caches"]
        tq.append_batch(caches, 0, state["k"], state["v"])
        first = caches[0].seq_length() - case["context"]
        return tq.compressed_attention(caches, 0, state["q"], start=first, use_qjl=case["qjl"])
    if kind == "window":
        state["window"].slide_window(state["k"], state["v"])
        return tq.hybrid_attention(state["cache"], state["window"], 0, state["q"])
    if kind == "prompt":
        n, heads, dim = case["tokens"], case["kv_heads"], case["dim"]
        cache = tq.TQKVCache(case["layers"], heads, dim)
        out = []
        for layer in range(case["layers"]):
            cache.append(layer, state["k"][layer], state["v"][layer])
        for layer in range(case["layers"]):
            k = torch.empty((n, heads, dim), device=DEV, dtype=torch.float16)
            v = torch.empty((n, heads, dim), device=DEV, dtype=torch.float16)
            cache.get_keys_fp16(layer, 0, n, out=k)
            cache.get_values_fp16(layer, 0, n, out=v)
            out.append((tq.compressed_attention(cache, layer, state["q"][layer], use_qjl=True), k, v))
        cache.close()
        return out
    n_out, n_in, w = case["out"], case["in"], state["w"]
    primary, residual = tq.fit_layer_codebooks(w, case["block"], 4, 4, 100)
    qw = tq.quantize_weight(w, primary, residual, tq.QuantizerConfig(4, 4, case["block"], case["shared"]))
    lin = tq.TurboQuantLinear(n_in, n_out, qw, primary, residual, case["block"])
    back = lin.dequantize(out=torch.empty((n_out, n_in), device=DEV, dtype=torch.float16))
    lin.close()
    return {"primary": primary.centroids, "residual": residual.centroids, "packed_primary": qw.packed_primary,
            "packed_residual": qw.packed_residual, "norms": qw.norms, "seeds": qw.seeds, "weights": back}


# ---- what a pass cannot do without -----------------------------------------------------------------------

# a stored token of one KV head: 3-bit codes in 32-bit words of ten for the key and the value, a norm for each, and
# the key's residual signs with their norm
def _token_bytes(dim, qjl):
    return 2 * (4 * -(-dim // 10) + 4) + ((4 * -(-dim // 32) + 4) if qjl else 0)


def _linear_work(n_in, n_out, rows, x_bytes=2, planes=1):
    return (n_in * n_out + 4 * n_out + rows * (x_bytes * n_in + 2 * n_out), 2 * planes * rows * n_in * n_out)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        b, f = _linear_work(case["in"], case["out"], case["rows"], 4 if case["host"] else 2, 1 if case["shared"] else 2)
        return {"bytes": case["layers"] * b, "flops": case["layers"] * f}
    if kind in ("project", "step"):
        rows, hidden, inter, dim = case["rows"], case["hidden"], case["inter"], case["dim"]
        q_out, kv_out = case["q_heads"] * dim, case["kv_heads"] * dim
        parts = [(hidden, q_out + 2 * kv_out), (q_out, hidden), (hidden, 2 * inter), (inter, hidden)]
        # activations between the projections could stay on the chip: only the layer's own ends count
        bytes_ = sum(i * o + 4 * o for i, o in parts) + rows * 2 * (2 * hidden + 2 * kv_out)
        flops = sum(2 * rows * i * o for i, o in parts)
        if kind == "project":
            bytes_ += rows * 2 * 2 * q_out
        else:
            bytes_ += rows * case["context"] * case["kv_heads"] * _token_bytes(dim, True)
            flops += rows * case["context"] * q_out * 6
        return {"bytes": bytes_, "flops": flops}
    if kind == "attend":
        tokens = case["seqs"] * case["context"]
        return {"bytes": tokens * case["kv_heads"] * _token_bytes(case["dim"], case["qjl"]) + case["seqs"] * case["q_heads"] * case["dim"] * 4,
                "flops": tokens * case["q_heads"] * case["dim"] * (6 if case["qjl"] else 4)}
    if kind == "window":
        return {"bytes": case["context"] * case["kv_heads"] * case["dim"] * 4 + case["q_heads"] * case["dim"] * 4,
                "flops": case["context"] * case["q_heads"] * case["dim"] * 4}
    if kind == "prompt":
        vectors = case["layers"] * case["tokens"] * case["kv_heads"]
        return {"bytes": vectors * (2 * case["dim"] * ((2 if case["f16"] else 4) + 2) + _token_bytes(case["dim"], True)),
                "flops": vectors * case["dim"] * 4 * int(math.log2(case["dim"]))}
    n = case["in"] * case["out"]
    return {"bytes": n * (4 + 1 + 2) + 4 * case["out"], "flops": 4 * n * int(math.log2(case["block"]))}


def tolerance(case):
    """fp16 rounds by up to 4.9e-4 of a value.  A linear rounds its input, its table and its result; a decoder layer
    chains six such steps.  Codes are whole numbers that a tie could move by one, which moves single weights."""
    kind = case["kind"]
    if kind == "linear":
        return {"rel": 1e-3}
    if kind in ("project", "step"):
        return {"rel": 2e-3}
    if kind in ("attend", "window", "prompt"):
        return {"rel": 1e-3}
    return {"rel": 1e-4, "max": 0.2, "differ": 1e-5}
