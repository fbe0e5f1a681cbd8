"""What a user of this package has it do: the workloads whose speed counts, through the public entry points.

Four kinds of work, each over the sizes that decoder models put through it:

* ``linear``   one ``QMatMul.forward``: decode (1 to 8 rows) and prefill (up to 2048 rows), any of the six weight
               formats, f32 / f16 / bf16 activations, with or without the prebuilt prefill image;
* ``layer``    the matmuls of one decode step of a decoder layer: grouped q|k|v, o, gate with SiLU on its store, up
               multiplied into it, down;
* ``experts``  one routed-expert projection (``QTensor.indexed_moe_forward``) of a batch of decode tokens;
* ``embed``    rows of a quantized embedding table for a batch of token ids (``QTensor.embedding``).

Weights are blocks of the package's own weight quantizer over N(0, 0.02) values: a pool of quantized blocks is made
from the seed and every block of a matrix is drawn from it, so that rows differ and large matrices are made quickly.
Activations are N(0, 1).
"""
from __future__ import annotations

import numpy as np
import torch

from lloom_b200 import GgmlDType, QMatMul, QTensor
from lloom_b200.quantized import forward_group, quantize_weights_host

DEVICE = "cuda"
FORMATS = ("Q4_0", "Q5_0", "Q8_0", "Q4K", "Q5K", "Q6K")
X_TYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _linear(name, fmt, m, n, k, x="f32", image=False):
    return {"name": name, "kind": "linear", "fmt": fmt, "m": m, "n": n, "k": k, "x": x, "image": image}


def listed():
    return [
        # the smallest call: a key / value projection of one decode token
        _linear("decode kv Q4_K m1", "Q4K", 1, 1024, 4096),
        # one decode token through a projection of a 2048-wide model
        _linear("decode Q8_0 m1", "Q8_0", 1, 8192, 2048),
        # one decode token through the output head, the largest matrix a model has
        _linear("lm_head Q6_K m1", "Q6K", 1, 128256, 4096),
        # eight sequences decoded together, gate / up projection
        _linear("decode Q4_K m8", "Q4K", 8, 14336, 4096),
        # an odd batch of sequences, the down projection as mixed-format files store it, bf16 hidden states
        _linear("decode Q6_K m5 bf16", "Q6K", 5, 4096, 14336, x="bf16"),
        # one decode token through the seven matmuls of a decoder layer (hidden 4096, 8 key / value heads)
        {"name": "layer Q4_K m1", "kind": "layer", "fmt": "Q4K", "m": 1, "hidden": 4096, "kv": 1024, "ffn": 14336},
        # a short prompt (or a batch of draft tokens), odd length, bf16 hidden states
        _linear("prompt Q5_K m37 bf16", "Q5K", 37, 4096, 4096, x="bf16"),
        # a medium prompt through an 8-bit model, f16 hidden states
        _linear("prefill Q8_0 m1000 f16", "Q8_0", 1000, 8192, 2048, x="f16"),
        # a prompt chunk through the down projection, prefill image kept beside the blocks
        _linear("prefill Q6_K m512 image", "Q6K", 512, 4096, 14336, image=True),
        # the largest: a long prompt chunk through the gate / up projection
        _linear("prefill Q4_K m2048", "Q4K", 2048, 14336, 4096),
        # four decode tokens through the gate projection of a mixture of experts
        {"name": "experts Q4_K b4 top8", "kind": "experts", "fmt": "Q4K", "experts": 64, "n": 1024, "k": 2048,
         "batch": 4, "topk": 8, "rows": 1},
        # a prompt's embeddings out of a 6-bit table
        {"name": "embed Q6_K 512 ids", "kind": "embed", "fmt": "Q6K", "n": 128256, "k": 4096, "ids": 512},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def _k_for(rng, fmt, lo, hi):
    """A row length the format has: whole 256-element blocks, or for the 32-element ones any multiple of 64."""
    step = 256 if fmt.endswith("K") else 64
    return max(step, _log_int(rng, lo, hi) // step * step)


def draw(rng):
    kind = rng.choices(("linear", "layer", "experts", "embed"), weights=(14, 2, 2, 1))[0]
    fmt = rng.choice(FORMATS)
    if kind == "linear":
        decode = rng.random() < 0.5
        m = rng.randint(1, 8) if decode else _log_int(rng, 9, 2048)
        n = _log_int(rng, 256, 32768) if decode else _log_int(rng, 256, 14336)
        k = _k_for(rng, fmt, 512, 14336)
        if decode:  # at most the output head's weights
            n = min(n, (1 << 28) // k)
        else:  # the formats with a scale per 32 elements have more to do per product
            limit = (1 << 36) if fmt.endswith("K") else (1 << 35)
            m = max(9, min(m, limit // (n * k)))
        return {"kind": kind, "fmt": fmt, "m": m, "n": n, "k": k, "x": rng.choice(("f32", "f32", "f16", "bf16")),
                "image": not decode and rng.random() < 0.3}
    if kind == "layer":
        hidden = _k_for(rng, fmt, 1024, 5120)
        return {"kind": kind, "fmt": fmt, "m": rng.randint(1, 8), "hidden": hidden, "kv": 64 * rng.randint(2, 16),
                "ffn": _k_for(rng, fmt, 2 * hidden, 4 * hidden)}
    if kind == "experts":
        topk = rng.randint(1, 8)
        return {"kind": kind, "fmt": fmt, "experts": rng.choice((8, 32, 64)), "n": _log_int(rng, 384, 2048),
                "k": _k_for(rng, fmt, 512, 4096), "batch": rng.randint(1, 8), "topk": topk, "rows": rng.choice((1, topk))}
    return {"kind": kind, "fmt": fmt, "n": _log_int(rng, 32000, 128256), "k": _k_for(rng, fmt, 1024, 4096),
            "ids": _log_int(rng, 1, 4096)}


# ---- inputs ----

def _weights(rng, fmt, shape):
    """A ``QTensor`` of ``shape`` on the GPU, its blocks drawn from a pool of quantized ones."""
    dtype = getattr(GgmlDType, fmt)
    be, bb = dtype.block_size(), dtype.type_size()
    pool = rng.standard_normal((512, 2048), dtype=np.float32) * np.float32(0.02)
    pool = torch.from_numpy(quantize_weights_host(pool, dtype).reshape(-1, bb))
    blocks = int(np.prod(shape, dtype=np.int64)) // be
    pick = torch.from_numpy(rng.integers(0, pool.shape[0], blocks, dtype=np.int32))
    return QTensor.from_data(torch.index_select(pool, 0, pick).reshape(-1), dtype, shape, DEVICE)


def _acts(gen, *shape, dtype=torch.float32):
    return torch.randn(*shape, generator=gen, device=DEVICE, dtype=torch.float32).to(dtype)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind, fmt = case["kind"], case["fmt"]
    state = {"case": case}
    if kind == "linear":
        w = _weights(rng, fmt, (case["n"], case["k"]))
        if case["image"]:
            w.storage.build_prefill_image(w.shape)
        state["mat"] = QMatMul.from_qtensor(w)
        state["x"] = _acts(gen, case["m"], case["k"], dtype=X_TYPES[case["x"]])
    elif kind == "layer":
        h, kv, f, m = case["hidden"], case["kv"], case["ffn"], case["m"]
        shapes = {"q": (h, h), "k": (kv, h), "v": (kv, h), "o": (h, h), "gate": (f, h), "up": (f, h), "down": (h, f)}
        state["mats"] = {name: QMatMul.from_qtensor(_weights(rng, fmt, s)) for name, s in shapes.items()}
        state["x"] = _acts(gen, m, h)        # normalized hidden state before the attention
        state["attn"] = _acts(gen, m, h)     # what the attention gives
        state["x_ffn"] = _acts(gen, m, h)    # normalized hidden state before the feed-forward
    elif kind == "experts":
        state["w"] = _weights(rng, fmt, (case["experts"], case["n"], case["k"]))
        state["x"] = _acts(gen, case["batch"], case["rows"], case["k"])
        scores = torch.rand(case["batch"], case["experts"], generator=gen, device=DEVICE)
        state["ids"] = scores.topk(case["topk"], dim=1).indices
    else:
        state["w"] = _weights(rng, fmt, (case["n"], case["k"]))
        state["ids"] = torch.randint(0, case["n"], (case["ids"],), generator=gen, device=DEVICE)
    return state


# ---- one pass ----

def run(state):
    kind = state["case"]["kind"]
    if kind == "linear":
        return state["mat"].forward(state["x"])
    if kind == "layer":
        w = state["mats"]
        q, k, v = forward_group([w["q"], w["k"], w["v"]], state["x"])
        o = w["o"].forward(state["attn"])
        h = w["gate"].forward_silu(state["x_ffn"])
        h = w["up"].forward_mul_into(state["x_ffn"], h)
        return q, k, v, o, h, w["down"].forward(h)
    if kind == "experts":
        return state["w"].indexed_moe_forward(state["x"], state["ids"])
    return state["w"].embedding(state["ids"])


# ---- what a pass cannot do without ----

def _packed(case, elems):
    dtype = getattr(GgmlDType, case["fmt"])
    return elems // dtype.block_size() * dtype.type_size()


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        size = X_TYPES[case["x"]].itemsize
        return {"bytes": _packed(case, n * k) + m * (n + k) * size, "flops": 2 * m * n * k}
    if kind == "layer":
        h, kv, f, m = case["hidden"], case["kv"], case["ffn"], case["m"]
        elems = 2 * h * h + 2 * kv * h + 3 * f * h
        # in: three hidden states; out: q, k, v, o, the gated product and the layer's output
        return {"bytes": _packed(case, elems) + 4 * m * (3 * h + 3 * h + 2 * kv + f), "flops": 2 * m * elems}
    if kind == "experts":
        n, k, e, b, t = case["n"], case["k"], case["experts"], case["batch"], case["topk"]
        distinct = e * (1 - (1 - t / e) ** b)  # experts that some token is routed to, on average
        return {"bytes": distinct * _packed(case, n * k) + 4 * b * (case["rows"] * k + t * n) + 8 * b * t,
                "flops": 2 * b * t * n * k}
    ids, k = case["ids"], case["k"]
    return {"bytes": ids * (_packed(case, k) + 4 * k + 8), "flops": ids * k}


def tolerance(case):
    if case["kind"] == "embed":
        return "exact"  # one element, one dequantization: no order to differ in
    x = case.get("x", "f32")
    if x == "f16":
        return {"rel": 1e-3, "max": 4e-3}
    if x == "bf16":
        return {"rel": 8e-3, "max": 3e-2}
    # Integer dots are exact; the f32 sums over the blocks of a row may be taken in any order.  A layer's last matmul
    # quantizes the product before it to 8 bits, and a value on the edge of two codes may fall to either side.
    return {"rel": 1e-3 if case["kind"] == "layer" else 1e-5}
