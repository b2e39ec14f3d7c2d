"""Timing cases: what a program that serves a quantized model has this framework do.

Four kinds of work, each through the public entry points that such a program calls:

  linear   one resident weight matrix times m activation rows (`DeviceWeights.gemv` / `.gemm`)
  layer    the linears of one or more decoder layers: q, k, v, o and the feed-forward block
           (`DeviceWeights.gemv` / `.gemm`, `device.ffn`), m tokens at a time
  moe      a mixture-of-experts feed-forward layer (`moe.MoeExperts.forward`)
  host     the kernel-trait call on host arrays (`KernelDispatcher.get_kernel(..).gemv` / `.gemm`),
           weights kept on the device by the library after their first use

Shapes are those of the repository's benchmark configurations (an 8B-class decoder layer in a
Q4_K / Q6_K mix, its LM head, a Q8_0 prefill matrix, an 8-expert MoE layer) and generic ones
around them.  Weights are random blocks with legal fields, activations N(0, 1).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from oxillama_b200 import moe as M
from oxillama_b200 import synth as S
from oxillama_b200.device import DeviceWeights, ffn
from oxillama_b200.kernels import KernelDispatcher, QuantTensor

TYPES = {name: t for t, name in S.NAMES.items()}
# per mix: the type of q, k, v, o, gate and up, and the type of down
MIXES = {"Q4_K_M": ("Q4_K", "Q6_K"), "Q5_K_M": ("Q5_K", "Q6_K"), "Q8_0": ("Q8_0", "Q8_0"), "Q4_0": ("Q4_0", "Q4_0"),
         "IQ4_XS": ("IQ4_XS", "IQ4_XS"), "Q3_K_M": ("Q3_K", "Q4_K"), "Q2_K": ("Q2_K", "Q3_K")}
# formats whose matmuls are computed with f32 operands at every batch size
F32_TYPES = ("Q5_K", "Q3_K", "Q2_K")


def _layer(name, mix, m, layers=1, hidden=4096, kv=1024, inter=14336):
    return {"name": name, "kind": "layer", "mix": mix, "hidden": hidden, "kv": kv, "inter": inter, "layers": layers, "m": m}


def _linear(name, qtype, rows, cols, m):
    return {"name": name, "kind": "linear", "type": qtype, "rows": rows, "cols": cols, "m": m}


def listed():
    return [
        # one K projection for one token: the smallest call of a decode step, all latency
        _linear("k_proj_q4k_m1", "Q4_K", 1024, 4096, 1),
        # one token through the linears of two layers: plain single-stream decoding
        _layer("decode_q4km_m1", "Q4_K_M", 1, layers=2),
        # the output head of that model, once per decoded token: the largest weight stream
        _linear("lm_head_q6k_m1", "Q6_K", 128256, 4096, 1),
        # decoding a model in the next larger K-quant mix
        _layer("decode_q5km_m1", "Q5_K_M", 1),
        # a handful of sequences decoded together
        _layer("batch_q4km_m8", "Q4_K_M", 8),
        # continuous batching: whatever number of sequences is live
        _layer("batch_q4km_m37", "Q4_K_M", 37),
        # a prompt of ordinary length
        _layer("prefill_q4km_m512", "Q4_K_M", 512),
        # a prompt whose length is no round number, on an 8-bit matrix
        _linear("prefill_q8_0_m509", "Q8_0", 4096, 4096, 509),
        # a long prompt chunk: the largest job
        _layer("prefill_q4km_m2048", "Q4_K_M", 2048),
        # three sequences decoded through an 8-expert layer, top-2
        {"name": "moe_decode_q4k_t3", "kind": "moe", "type": "Q4_K", "hidden": 4096, "inter": 14336, "experts": 8, "top_k": 2,
         "tokens": 3},
        # a prompt of 256 tokens through the same layer in the non-linear 4-bit format
        {"name": "moe_prefill_iq4xs_t256", "kind": "moe", "type": "IQ4_XS", "hidden": 4096, "inter": 14336, "experts": 8,
         "top_k": 2, "tokens": 256},
        # the trait call of a host program: slices in, slice out, one token at the FFN-up shape
        {"name": "host_q4k_m1", "kind": "host", "type": "Q4_K", "rows": 14336, "cols": 4096, "m": 1},
    ]


# ------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, step):
    return max(step, _log(rng, lo, hi) // step * step)


def _matrix(rng, qtype, max_rows, max_cols):
    rows = _log(rng, 256, max_rows)
    if rng.random() < 0.6:
        rows = max(64, rows // 64 * 64)
    # rows are whole blocks: 32 columns for the 32-weight formats, 256 for the super-block ones
    step = 32 if qtype in ("Q4_0", "Q8_0") and rng.random() < 0.4 else 256
    return rows, _size(rng, 512, max_cols, step)


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "layer", "layer", "moe", "moe", "host"])
    main = ["Q4_K", "Q4_K", "Q6_K", "Q8_0", "Q4_0", "IQ4_XS"]
    if kind == "linear":
        qtype = rng.choice(main + list(F32_TYPES[:2]))
        few = qtype in F32_TYPES
        m = _log(rng, 1, 4 if few else 2048)
        if m <= 4 and not few and rng.random() < 0.2:
            rows, cols = _log(rng, 32000, 128256), _size(rng, 2048, 4096, 256)  # an output head
        else:
            rows, cols = _matrix(rng, qtype, 14336, 14336)
        return {"kind": kind, "type": qtype, "rows": rows, "cols": cols, "m": m}
    if kind == "layer":
        mix = rng.choice(["Q4_K_M", "Q4_K_M", "Q5_K_M", "Q8_0", "Q4_0", "IQ4_XS", "Q3_K_M"])
        few = any(t in F32_TYPES for t in MIXES[mix])
        hidden = _size(rng, 1024, 4096, 256)
        return {"kind": kind, "mix": mix, "hidden": hidden, "kv": hidden // 4, "inter": min(14336, _size(rng, 2 * hidden, 3.5 * hidden, 256)),
                "layers": 1, "m": _log(rng, 1, 4 if few else 2048)}
    if kind == "moe":
        hidden = _size(rng, 1024, 4096, 256)
        experts = rng.choice([4, 8, 8, 16])
        return {"kind": kind, "type": rng.choice(["Q4_K", "IQ4_XS", "Q8_0", "Q6_K"]), "hidden": hidden,
                "inter": _size(rng, hidden, 3.5 * hidden if experts <= 8 else 1.5 * hidden, 256), "experts": experts,
                "top_k": rng.choice([1, 2, 2, 3]), "tokens": _log(rng, 1, 512)}
    qtype = rng.choice(main)
    rows, cols = _matrix(rng, qtype, 14336, 8192)
    return {"kind": kind, "type": qtype, "rows": rows, "cols": cols, "m": _log(rng, 1, 64)}


# ------------------------------------------------------------------ inputs
def _blocks(gen, qtype, rows, cols):
    """Random blocks of `rows` rows as host bytes.  Every field but the scales may hold any
    value; f16 scales are uniform, Q6_K's int8 sub-scales lie in [-32, 31]."""
    bb = S.BLOCK_BYTES[qtype]
    n = rows * S.blocks_per_row(qtype, cols)
    b = torch.randint(0, 256, (n, bb), dtype=torch.uint8, device="cuda", generator=gen)

    def f16(at, lo=1e-4, hi=2e-3):
        v = torch.empty(n, dtype=torch.float32, device="cuda").uniform_(lo, hi, generator=gen)
        b[:, at:at + 2] = v.half().view(torch.uint8).view(n, 2)

    if qtype in (S.Q4_0, S.Q8_0, S.IQ4_XS):
        f16(0)
    elif qtype in (S.Q4_K, S.Q5_K):
        f16(0)
        f16(2)
    elif qtype == S.Q6_K:
        b[:, 192:208] = torch.randint(-32, 32, (n, 16), dtype=torch.int8, device="cuda", generator=gen).view(torch.uint8)
        f16(208)
    elif qtype == S.Q3_K:
        f16(108)
    elif qtype == S.Q2_K:
        f16(80)
        f16(82)
    return b.view(-1).cpu().numpy()


def _weights(gen, qtype, rows, cols):
    return DeviceWeights(qtype, _blocks(gen, qtype, rows, cols), rows, cols)


def _acts(gen, *shape):
    return torch.randn(shape, device="cuda", generator=gen)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "linear":
        t, rows, cols, m = TYPES[case["type"]], case["rows"], case["cols"], case["m"]
        st.update(w=_weights(gen, t, rows, cols), x=_acts(gen, m, cols), y=torch.empty(m, rows, device="cuda"), m=m)
    elif kind == "layer":
        ta, tb = (TYPES[t] for t in MIXES[case["mix"]])
        h, kv, inter, m = case["hidden"], case["kv"], case["inter"], case["m"]
        st["m"], st["layers"] = m, []
        for _ in range(case["layers"]):
            lw = [_weights(gen, ta, r, h) for r in (h, kv, kv, h)]  # q, k, v, o
            fw = [_weights(gen, ta, inter, h), _weights(gen, ta, inter, h), _weights(gen, tb, h, inter)]  # gate, up, down
            xs = [_acts(gen, m, h) for _ in range(3)]  # into q, k, v; into o; into the feed-forward block
            ys = [torch.empty(m, r, device="cuda") for r in (h, kv, kv, h, h)]
            st["layers"].append((lw, fw, xs, ys))
    elif kind == "moe":
        t, h, inter, n = TYPES[case["type"]], case["hidden"], case["inter"], case["experts"]
        # Two seeded draws per projection, dealt to the experts in turn and each uploaded as a
        # matrix of its own: the sizes and the traffic of independent experts.
        g, u, d = ([_blocks(gen, t, r, c) for _ in range(2)] for r, c in ((inter, h), (inter, h), (h, inter)))
        st["experts"] = M.MoeExperts(t, [g[e % 2] for e in range(n)], [u[e % 2] for e in range(n)], [d[e % 2] for e in range(n)],
                                     h, inter, n)
        st.update(logits=_acts(gen, case["tokens"], n), x=_acts(gen, case["tokens"], h),
                  y=torch.empty(case["tokens"], h, device="cuda"), top_k=case["top_k"])
    else:
        t, rows, cols, m = TYPES[case["type"]], case["rows"], case["cols"], case["m"]
        st.update(kernel=KernelDispatcher().get_kernel(t), w=QuantTensor(_blocks(gen, t, rows, cols), (rows, cols), t),
                  x=_acts(gen, m, cols).cpu().numpy(), y=np.empty((m, rows), np.float32), m=m, rows=rows, cols=cols)
    return st


# ------------------------------------------------------------------ one pass
def _matmul(w, x, y, m):
    if m == 1:
        w.gemv(x, y)
    else:
        w.gemm(x, y, m)


def run(st):
    kind = st["kind"]
    if kind == "linear":
        _matmul(st["w"], st["x"], st["y"], st["m"])
        return st["y"]
    if kind == "layer":
        m = st["m"]
        for (wq, wk, wv, wo), (wg, wu, wd), (x0, x1, x2), (yq, yk, yv, yo, yf) in st["layers"]:
            _matmul(wq, x0, yq, m)
            _matmul(wk, x0, yk, m)
            _matmul(wv, x0, yv, m)
            _matmul(wo, x1, yo, m)
            ffn(wg, wu, wd, x2, yf, m)
        return [layer[3] for layer in st["layers"]]
    if kind == "moe":
        st["experts"].forward(st["logits"], st["x"], st["y"], st["top_k"])
        return st["y"]
    if st["m"] == 1:
        st["kernel"].gemv(st["w"], st["x"], st["y"])
    else:
        st["kernel"].gemm(st["w"], st["x"], st["y"], st["m"], st["rows"], st["cols"])
    return st["y"]


# ------------------------------------------------------------------ work and tolerance
def _matrices(case):
    """(type name, rows, cols, times) of the matrices that one pass multiplies by `m` rows each."""
    if case["kind"] == "layer":
        ta, tb = MIXES[case["mix"]]
        h, kv, inter = case["hidden"], case["kv"], case["inter"]
        return [(ta, h, h, 2), (ta, kv, h, 2), (ta, inter, h, 2), (tb, h, inter, 1)]
    return [(case["type"], case["rows"], case["cols"], 1)]


def work(case):
    if case["kind"] == "moe":
        h, inter, n, k, t = case["hidden"], case["inter"], case["experts"], min(case["top_k"], case["experts"]), case["tokens"]
        q = TYPES[case["type"]]
        per_expert = 2 * S.weight_nbytes(q, inter, h) + S.weight_nbytes(q, h, inter)
        hit = n * (1.0 - (1.0 - k / n) ** t)  # experts that get a token, on average
        return {"bytes": hit * per_expert + 4.0 * t * (2 * h + n), "flops": 2.0 * t * k * 3 * h * inter}
    m, nbytes, flops = case["m"], 0.0, 0.0
    for t, rows, cols, times in _matrices(case):
        nbytes += times * S.weight_nbytes(TYPES[t], rows, cols)
        flops += times * 2.0 * m * rows * cols
    if case["kind"] == "layer":  # three inputs and five outputs; what lies between gate / up and down stays inside
        nbytes += 4.0 * m * (6 * case["hidden"] + 2 * case["kv"])
    else:
        nbytes += 4.0 * m * (case["rows"] + case["cols"])
    layers = case.get("layers", 1)
    return {"bytes": layers * nbytes, "flops": layers * flops}


def tolerance(case):
    # Up to four rows (two of Q6_K) and the formats without a matrix-unit path are f32-grade sums;
    # larger batches multiply 16-bit operands (f32 sums): 2^-11 per operand, averaged over a row.
    if case["kind"] == "moe":
        types, m = [case["type"]], case["tokens"]
    else:
        types, m = [t for t, *_ in _matrices(case)], case["m"]
    half = any(t not in F32_TYPES and m > (2 if t == "Q6_K" else 4) for t in types)
    return {"rel": 1e-3, "max": 1e-2} if half else {"rel": 2e-5, "max": 2e-4}
