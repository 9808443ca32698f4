"""What a program that uses this framework has it do, as cases that can be timed and compared.

A case names an operation ("op"), the block format and the sizes; `prepare` makes the coded weights and the inputs,
`run` makes one pass through the public entry points.  The operations:

  linear   CodedMatrix.linear: y[m, N] = x[m, K] . W^T, activations and result on the GPU
  batch    ProductBatch: several one-row products that read the same activations (gate and up; q, k and v)
  host     CodedMatrix.matmul: the same product on host arrays (rt_test_matmul)
  weights  CodedMatrix.decode_weights: the whole matrix as fp16 on the GPU
  codes    CodedMatrix.decode_codes: the whole matrix as one code per byte on the GPU
  codec    bundle.encode_huf8 and bundle.decode_huf8 on host arrays
  decoder  Bundle.forward on a whole model: `tokens` tokens that follow `context` tokens already in the KV cache

Codes and scales follow lazyweights_b200.modelgen; the scales are smaller and the offsets sit at the codes' centre, so
that a decoder's activations stay in the range that they have in a trained model.
"""
import ctypes as C
import math
import tempfile

import numpy as np
import torch

import lazyweights_b200 as lw
from lazyweights_b200.bundle import ROPE_ROWS, Writer
from lazyweights_b200.modelgen import MISTRAL_7B, PHI3_MINI, SIDE_BYTES

PAIRED = ("Q4_K", "IQ4_XS")
FORMATS = ("Q4_K", "Q5_K", "Q6_K", "IQ4_XS")
SHAPES = {"mistral": MISTRAL_7B, "phi3": PHI3_MINI}
CENTRE = {"Q4_K": 8.0, "IQ4_XS": 7.5, "Q5_K": 16.0, "Q6_K": 32.0}
TOP = {"Q4_K": 15, "IQ4_XS": 15, "Q5_K": 31, "Q6_K": 63}
# fp16 super-block scale at which the weights' standard deviation is about 0.02
SCALE = {"Q4_K": 2.6e-4, "Q5_K": 2.2e-4, "Q6_K": 1.1e-4, "IQ4_XS": 4e-5}
# entropy of the code distributions below, bits per weight: what a coded weight takes at least
ENTROPY = {"Q4_K": 3.02, "IQ4_XS": 3.02, "Q5_K": 3.37, "Q6_K": 4.37}


def listed():
    return [
        # the smallest call: the k (or v) projection of one token, grouped-query attention
        dict(name="kv_row_q5k", op="linear", fmt="Q5_K", N=1024, K=4096, m=1, half=True),
        # one token through an attention projection
        dict(name="attn_row_q4k", op="linear", fmt="Q4_K", N=4096, K=4096, m=1, half=True),
        # one token through gate and up of a feed-forward block, one launch
        dict(name="ffn_pair_q6k", op="batch", fmt="Q6_K", N=14336, K=4096, count=2, half=True),
        # a caller of the reference's entry point, activations and result in host memory
        dict(name="host_row_iq4xs", op="host", fmt="IQ4_XS", N=8192, K=3072, m=1),
        # eight rows: a small batch, or the verification of drafted tokens
        dict(name="ffn_rows8_q6k", op="linear", fmt="Q6_K", N=14336, K=4096, m=8, half=True),
        # a decode batch of an odd size, fp32 activations as the decoder runtime has them
        dict(name="attn_rows33_q5k", op="linear", fmt="Q5_K", N=4096, K=4096, m=33, half=False),
        # a prompt through the largest projection
        dict(name="ffn_rows512_q4k", op="linear", fmt="Q4_K", N=14336, K=4096, m=512, half=True),
        # weights for a caller's own kernels, or a check against another dequantiser
        dict(name="weights_q4k", op="weights", fmt="Q4_K", N=4096, K=14336),
        # building a bundle and reading a tensor of it back
        dict(name="codec_q5k", op="codec", fmt="Q5_K", N=4096, K=4096),
        # batch-1 decoding at a context of 2048: one token
        dict(name="decoder_token", op="decoder", shape="mistral", fmt="Q4_K", ffn="Q4_K", layers=32, vocab=32000,
             context=2047, tokens=1, every=False),
        # speculative decoding: the last token and seven drafts verified in one pass
        dict(name="decoder_verify", op="decoder", shape="phi3", fmt="IQ4_XS", ffn="IQ4_XS", layers=32, vocab=32064,
             context=1000, tokens=8, every=True),
        # a prompt of 128 tokens into an empty cache
        dict(name="decoder_prompt", op="decoder", shape="mistral", fmt="Q4_K", ffn="Q4_K", layers=32, vocab=32000,
             context=0, tokens=128, every=False),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi, unit):
    """A multiple of `unit`, spread over the logarithm of the range."""
    return max(lo, min(hi, int(round(_log(rng, lo, hi) / unit)) * unit))


def _matrix(rng, fmt):
    while True:
        n, k = _size(rng, 256, 14336, 64), _size(rng, 512, 14336, 512 if fmt in PAIRED else 256)
        if n * k <= 14336 * 4096:
            return n, k


def draw(rng):
    op = rng.choices(("linear", "batch", "host", "weights", "codes", "codec", "decoder"), (10, 3, 2, 2, 2, 1, 2))[0]
    fmt = rng.choice(FORMATS)
    n, k = _matrix(rng, fmt)
    if op == "linear":
        return dict(op=op, fmt=fmt, N=n, K=k, m=int(round(_log(rng, 1, 512))), half=rng.random() < 0.5)
    if op == "batch":
        return dict(op=op, fmt=fmt, N=n, K=k, count=rng.randint(2, 3 if n * k < 2e7 else 2), half=rng.random() < 0.5)
    if op == "host":
        return dict(op=op, fmt=fmt, N=n, K=k, m=int(round(_log(rng, 1, 16))))
    if op in ("weights", "codes"):
        return dict(op=op, fmt=fmt, N=n, K=k)
    if op == "codec":
        return dict(op=op, fmt=fmt, N=min(n, 4096), K=min(k, 4096))
    context = int(round(_log(rng, 16, 2048)))
    return dict(op=op, shape=rng.choice(("mistral", "phi3")), fmt=fmt, ffn=rng.choice(FORMATS), layers=rng.randint(2, 6),
                vocab=_size(rng, 4096, 32000, 64), context=context, tokens=int(round(_log(rng, 1, 160))),
                every=rng.random() < 0.3)


# ------------------------------------------------------------------------------------------------------- inputs


def _codes(fmt, n, k, gen):
    """uint8 codes [n, k] on the GPU: discretised Laplace (4-bit formats) or Gaussian."""
    if fmt in PAIRED:
        x = torch.empty((n, k), device="cuda").exponential_(generator=gen)
        x -= torch.empty((n, k), device="cuda").exponential_(generator=gen)
        x *= 1.5
    else:
        x = torch.randn((n, k), device="cuda", generator=gen)
        x *= 2.5 if fmt == "Q5_K" else 5.0
    return x.add_(CENTRE[fmt]).round_().clamp_(0, TOP[fmt]).to(torch.uint8)


def _symbols(fmt, n, k, gen):
    q = _codes(fmt, n, k, gen)
    return (q[:, 0::2] | (q[:, 1::2] << 4)).cpu().numpy() if fmt in PAIRED else q.cpu().numpy()


def _side(fmt, n, k, rng):
    nb = n * k // 256
    side = rng.integers(0, 256, (nb, SIDE_BYTES[fmt]), dtype=np.uint8)
    d = (SCALE[fmt] * rng.uniform(0.5, 1.5, nb)).astype(np.float16)
    if fmt in ("Q4_K", "Q5_K"):   # the minimum of a sub-block is its scale times the centre of the codes
        side[:, 0:2] = d.view(np.uint8).reshape(nb, 2)
        side[:, 2:4] = (d * np.float16(CENTRE[fmt])).view(np.uint8).reshape(nb, 2)
        side[:, 8:12] = side[:, 4:8]
        side[:, 12:16] = (side[:, 12:16] & 15) * 17
    elif fmt == "Q6_K":
        side[:, 0:16] = rng.integers(-64, 64, (nb, 16)).astype(np.int8).view(np.uint8)
        side[:, 16:18] = d.view(np.uint8).reshape(nb, 2)
    else:
        side[:, 0:2] = d.view(np.uint8).reshape(nb, 2)
    return side.reshape(n, -1)


def _most(sym):
    """The bytes that a blob of these symbols can take: table, lane offsets, 11 bits a symbol, tail."""
    return 4096 + sym.size // 128 + sym.size * 11 // 8 + 16


def _encode(sym):
    """The blob of symbols [N, Ks], by the library's encoder."""
    n, ks = sym.shape
    out = np.empty(_most(sym), np.uint8)
    bits = C.c_longlong(0)
    size = lw.lib().lw_encode_huf8(sym.ctypes.data, n, ks, out.ctypes.data, out.size, C.byref(bits))
    assert 0 < size <= out.size
    return out[:size]


def _generators(seed):
    return torch.Generator(device="cuda").manual_seed(seed), np.random.default_rng(seed)


def _coded(fmt, n, k, gen, rng):
    sym = _symbols(fmt, n, k, gen)
    return lw.CodedMatrix(_encode(sym), n, sym.shape[1], fmt, _side(fmt, n, k, rng))


def _activations(m, k, half, gen):
    x = torch.randn((m, k), device="cuda", generator=gen)
    return x.half() if half else x


def _bundle(case, seed):
    """A random model of the case's shape, written as a bundle and opened; the layers share the bytes in the file, on
    the GPU every layer has its own."""
    gen, rng = _generators(seed)
    s = SHAPES[case["shape"]]
    d, h, hk, dh, inter = s["hidden"], s["n_heads"], s["n_kv_heads"], s["head_dim"], s["inter"]
    layers, vocab = case["layers"], case["vocab"]
    tokens, context = case["tokens"], case["context"]
    with tempfile.TemporaryDirectory() as path:
        w = Writer(path)
        for key, v in dict(n_layers=layers, hidden=d, n_heads=h, n_kv_heads=hk, head_dim=dh, inter=inter, vocab=vocab,
                           eps=s["eps"], rope_rows=ROPE_ROWS, rope_half=dh // 2, attn_scale=dh ** -0.5, enc="kq_huf",
                           tied=0, eos="2").items():
            w.cfg(key, v)
        embed = (torch.randn((vocab, d), device="cuda", generator=gen) * 0.05).half().cpu().numpy()
        w.add("embed", "f16", vocab, d, 1.0, 0, embed.reshape(-1).view(np.uint8).data)
        inv = 1.0 / (s["theta"] ** (np.arange(0, dh, 2, dtype=np.float64) / dh))
        angle = np.arange(ROPE_ROWS, dtype=np.float64)[:, None] * inv[None]
        w.add("cos", "f32", ROPE_ROWS, dh // 2, 1.0, 0, np.cos(angle).astype(np.float32).tobytes())
        w.add("sin", "f32", ROPE_ROWS, dh // 2, 1.0, 0, np.sin(angle).astype(np.float32).tobytes())
        for name in ["l%d.ln%d" % (i, j) for i in range(layers) for j in (1, 2)] + ["lnf"]:
            w.add(name, "f32", 1, d, 1.0, 0, (1.0 + 0.1 * rng.standard_normal(d)).astype(np.float32).tobytes())
        for name, fmt, n, k, copies in (("qkv", case["fmt"], (h + 2 * hk) * dh, d, layers), ("o", case["fmt"], d, h * dh, layers),
                                        ("gate", case["ffn"], inter, d, layers), ("up", case["ffn"], inter, d, layers),
                                        ("down", case["ffn"], d, inter, layers), ("lm_head", case["fmt"], vocab, d, 0)):
            first = len(w.lines)
            name0 = "l0." + name if copies else name
            side = _side(fmt, n, k, rng)
            w.add(name0, "huf4p" if fmt in PAIRED else "huf8", n, k, 1.0, 0, _encode(_symbols(fmt, n, k, gen)).data)
            w.add(name0 + ".kqs", "kq_" + fmt, n, side.shape[1], 1.0, 0, side.reshape(-1).data)
            for line in w.lines[first:]:
                w.lines += [line.replace(" l0.", " l%d." % i, 1) for i in range(1, copies)]
        w.close()
        b = lw.Bundle(path, max_ctx=ROPE_ROWS, max_batch=max(64, tokens))
    ids = rng.integers(0, vocab, context + tokens)
    if context:
        b.forward(ids[:context])
    return b, np.ascontiguousarray(ids[context:], np.int32)


def prepare(case, seed):
    op = case["op"]
    if op == "decoder":
        b, ids = _bundle(case, seed)
        return dict(case=case, bundle=b, ids=ids)
    gen, rng = _generators(seed)
    fmt, n, k = case["fmt"], case["N"], case["K"]
    if op == "codec":
        sym = _symbols(fmt, n, k, gen)
        return dict(case=case, sym=sym, blob=np.zeros(_most(sym), np.uint8))
    if op == "batch":
        mats = [_coded(fmt, n, k, gen, rng) for _ in range(case["count"])]
        x = _activations(1, k, case["half"], gen)[0]
        ys = [torch.empty(n, device="cuda") for _ in mats]
        return dict(case=case, mats=mats, ys=ys, batch=lw.ProductBatch([(a, a.NAME, x, y) for a, y in zip(mats, ys)]))
    st = dict(case=case, mat=_coded(fmt, n, k, gen, rng))
    if op == "linear":
        st["x"] = _activations(case["m"], k, case["half"], gen)
        st["y"] = torch.empty((case["m"], n), device="cuda")
    elif op == "host":
        st["x"] = rng.standard_normal((case["m"], k), dtype=np.float32)
    elif op == "weights":
        st["out"] = torch.empty((n, k), dtype=torch.float16, device="cuda")
    else:
        st["out"] = torch.empty((n, k), dtype=torch.uint8, device="cuda")
    return st


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "linear":
        return state["mat"].linear(lw.CodedMatrix.NAME, state["x"], out=state["y"])
    if op == "batch":
        state["batch"].launch()
        return state["ys"]
    if op == "host":
        return state["mat"].matmul(lw.CodedMatrix.NAME, state["x"])
    if op == "weights":
        return state["mat"].decode_weights(lw.CodedMatrix.NAME, out=state["out"])
    if op == "codes":
        return state["mat"].decode_codes(lw.CodedMatrix.NAME, out=state["out"])
    if op == "codec":
        sym, out = state["sym"], state["blob"]
        blob, bits, hist = lw.bundle.encode_huf8(sym)
        out[:len(blob)] = np.frombuffer(blob, np.uint8)   # a buffer of one size for blobs of any
        return [out, bits, hist, lw.bundle.decode_huf8(blob, *sym.shape)]
    b = state["bundle"]
    b.set_pos(case["context"])
    return b.forward(state["ids"], all_logits=case["every"])


# --------------------------------------------------------------------------------------------- work and tolerance


def _matrix_bytes(fmt, n, k):
    """Coded weights, side bytes."""
    return n * k * ENTROPY[fmt] / 8 + n * k // 256 * SIDE_BYTES[fmt]


def work(case):
    op = case["op"]
    if op == "decoder":
        s = SHAPES[case["shape"]]
        d, h, hk, dh, inter, t = s["hidden"], s["n_heads"], s["n_kv_heads"], s["head_dim"], s["inter"], case["tokens"]
        span = case["context"] + t
        rows = t if case["every"] else 1
        attn, ffn = (h + 2 * hk) * dh * d + d * h * dh, 3 * inter * d
        layer = _matrix_bytes(case["fmt"], 1, attn) + _matrix_bytes(case["ffn"], 1, ffn) + 2 * hk * dh * span * 2
        head = _matrix_bytes(case["fmt"], case["vocab"], d) + rows * case["vocab"] * 4 + t * d * 2
        flops = case["layers"] * (2 * t * (attn + ffn) + 4 * h * dh * t * (case["context"] + (t + 1) / 2)) + 2 * rows * case["vocab"] * d
        return {"bytes": case["layers"] * layer + head, "flops": flops}
    fmt, n, k = case["fmt"], case["N"], case["K"]
    if op == "weights":
        return {"bytes": _matrix_bytes(fmt, n, k) + 2 * n * k, "flops": 0}
    if op == "codes":
        return {"bytes": n * k * ENTROPY[fmt] / 8 + n * k, "flops": 0}
    if op == "codec":
        ks = k // 2 if fmt in PAIRED else k
        return {"bytes": 2 * n * ks + 2 * n * k * ENTROPY[fmt] / 8, "flops": 0}
    m, count = case.get("m", 1), case.get("count", 1)
    x = m * k * (2 if case.get("half") else 4)
    return {"bytes": count * (_matrix_bytes(fmt, n, k) + m * n * 4) + x, "flops": 2 * m * n * k * count}


def tolerance(case):
    op = case["op"]
    if op in ("weights", "codes", "codec"):
        return "exact"
    if op == "decoder":   # fp16 KV cache; fp16 operands in passes of more than eight tokens; errors of all layers
        return {"rel": 1e-2}
    if case.get("m", 1) <= 8:   # activations in 16-bit fixed point per sub-block, fp32 sums
        return {"rel": 1e-4}
    return {"rel": 2e-3}        # fp16 weights and activations, fp32 sums
