"""Performance cases: the work that a program built on this package has it do, at sizes of the
decoder shapes in lutmac_b200/synth.py.

Families (`"op"` of a case):
  linear    Context.linear on resident weights and device buffers, every block kind, batch 1 to 32
  group     Group.launch: all projections of some decoder layers as one prepared launch
  host      api.lut_linear, the reference's layer call: host arrays in, host array out
  quantize  api.quantize_tensor: an fp32 matrix into the blocks of a checkpoint
  decode    Model.forward on consecutive positions: single-token decode, batched decode, prompts
"""
import math

import numpy as np
import torch

from lutmac_b200 import synth
from lutmac_b200.api import Group, default_context, lut_linear, quantize_tensor
from lutmac_b200.blocks import (BINARY, BLOCK_BYTES, BLOCK_DTYPES, DEFAULT_QUANT_BITS, INT2, INT3, INT4, INT5, INT6, INT8,
                                KIND_NAMES, TERNARY, PackedTensor, algorithmic_bytes, blocks_per_row)
from lutmac_b200.model import Model

KINDS = {name: kind for kind, name in KIND_NAMES.items()}
MAX_SEQ = 2048  # cache positions per sequence, the reference's default
DEVICE = "cuda:0"


# ---- the cases ------------------------------------------------------------------------------------------

def listed():
    return [
        # the smallest call in use: one ternary q projection of a 1B decoder, latency only
        dict(name="linear_ternary_2048x2048", op="linear", kind="ternary", M=2048, K=2048, batch=1, bias=False),
        # sizes that divide by nothing, with a bias (imported checkpoints with odd widths), few rows
        dict(name="linear_int3_1001x1500_bias", op="linear", kind="int3", M=1001, K=1500, batch=1, bias=True),
        # the vocabulary projection of a 1B decoder, which every model here keeps in 8 bits
        dict(name="linear_int8_128256x2048", op="linear", kind="int8", M=128256, K=2048, batch=1, bias=False),
        # a feed-forward down projection of a 70B decoder for 16 sequences
        dict(name="linear_ternary_8192x28672_b16", op="linear", kind="ternary", M=8192, K=28672, batch=16, bias=False),
        # the seven 4-bit projections of eight 1B layers prepared once and issued together
        dict(name="group_int4_1b_8_layers", op="group", shape="llama-3.2-1b", kind="int4", layers=8),
        # the reference's own layer call on host arrays: 2-bit gate projection, 4 sequences, with bias
        dict(name="host_int2_8960x1536_b4", op="host", kind="int2", M=8960, K=1536, batch=4, bias=True),
        # making a checkpoint: one 4-bit gate projection of a 1B decoder
        dict(name="quantize_int4_8192x2048", op="quantize", kind="int4", M=8192, K=2048, rotate=False),
        # interactive decode of the whole 1B decoder: every token's logits go to the sampler on the host
        dict(name="decode_1b_int4_b1", op="decode", shape="llama-3.2-1b", kind="int4", layers=16, vocab=128256, batch=1,
             context=512, steps=4, logits="every"),
        # a prompt: positions from 0, only the last token's logits are wanted
        dict(name="prompt_1b_int4_24_tokens", op="decode", shape="llama-3.2-1b", kind="int4", layers=16, vocab=128256,
             batch=1, context=0, steps=24, logits="last"),
        # serving a 1.5B decoder in 2-bit residual form with biases to 32 sequences (8 of its 28 layers)
        dict(name="decode_1.5b_int2_b32", op="decode", shape="qwen-2.5-1.5b", kind="int2", layers=8, vocab=151936,
             batch=32, context=1024, steps=2, logits="every"),
        # the 70B-shaped ternary stack, one and 16 sequences over a long context (4 of its 80 layers, and
        # a vocabulary that leaves the head about the share of a step that it has with all layers)
        dict(name="decode_70b_ternary_b1", op="decode", shape="llama-3-70b", kind="ternary", layers=4, vocab=16384, batch=1,
             context=2040, steps=2, logits="every"),
        dict(name="decode_70b_ternary_b16", op="decode", shape="llama-3-70b", kind="ternary", layers=4, vocab=16384, batch=16,
             context=2040, steps=2, logits="every"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A width or height: a multiple of 256 as often as any other number."""
    n = _log_int(rng, lo, hi)
    return max(256, n // 256 * 256) if rng.random() < 0.5 else n


def _batch(rng, most):
    return 1 if rng.random() < 0.4 else _log_int(rng, 2, most)


def _draw_any(rng):
    op = rng.choice(["linear", "linear", "linear", "decode", "decode", "decode", "group", "host", "quantize"])
    if op in ("linear", "host"):
        c = dict(op=op, kind=rng.choice(sorted(KINDS)), M=_size(rng, 64, 32768), K=_size(rng, 64, 28672),
                 batch=_batch(rng, 32), bias=rng.random() < 0.3)
        if op == "host":
            c["M"], c["K"] = min(c["M"], 16384), min(c["K"], 8192)
        return c
    if op == "quantize":
        kind = rng.choice(["ternary", "binary", "int2", "int3", "int4", "int8"])
        return dict(op=op, kind=kind, M=_size(rng, 64, 8192), K=_size(rng, 64, 4096),
                    rotate=kind in ("ternary", "binary", "int2"))
    if op == "group":
        return dict(op=op, shape=rng.choice(["llama-3.2-1b", "qwen-2.5-1.5b"]), kind=rng.choice(["ternary", "int2", "int4", "int8"]),
                    layers=rng.randint(1, 8))
    shape = rng.choice(sorted(synth.MODEL_SHAPES))
    large = shape == "llama-3-70b"
    batch = _batch(rng, 16 if large else 32)
    return dict(op=op, shape=shape, kind=rng.choice(["ternary", "int2", "int3", "int4", "int8"]),
                layers=rng.randint(1, 2) if large else rng.randint(2, 8), vocab=_log_int(rng, 4096, 32768) if large else 32000,
                batch=batch, context=_log_int(rng, 1, 2040) if rng.random() < 0.9 else 0, steps=rng.randint(1, 8),
                logits=rng.choice(["every", "last"]))


def draw(rng):
    most = {k: max(work(c)[k] for c in listed()) for k in ("bytes", "flops")}
    while True:
        c = _draw_any(rng)
        w = work(c)
        if w["bytes"] <= most["bytes"] and w["flops"] <= most["flops"]:
            return c


# ---- what a pass cannot do without ------------------------------------------------------------------------

def _projections(shape):
    h, it, hd = shape["hidden"], shape["inter"], shape["head_dim"]
    qd, kvd = shape["n_heads"] * hd, shape["n_kv_heads"] * hd
    return [("q", qd, h), ("k", kvd, h), ("v", kvd, h), ("o", h, qd), ("gate", it, h), ("up", it, h), ("down", h, it)]


def work(case):
    op, kind = case["op"], KINDS[case["kind"]]
    if op in ("linear", "host"):
        M, K, b = case["M"], case["K"], case["batch"]
        return {"bytes": M * blocks_per_row(K) * BLOCK_BYTES[kind] + 4 * b * (K + M) + (4 * M if case["bias"] else 0),
                "flops": 2 * M * K * b}
    if op == "quantize":
        M, K = case["M"], case["K"]
        return {"bytes": 4 * M * K + M * blocks_per_row(K) * BLOCK_BYTES[kind], "flops": 4 * M * K}
    shape = synth.MODEL_SHAPES[case["shape"]]
    if op == "group":
        p = [(M, K) for _, M, K in _projections(shape)]
        return {"bytes": case["layers"] * sum(algorithmic_bytes(kind, M, K) for M, K in p),
                "flops": case["layers"] * sum(2 * M * K for M, K in p)}
    b, steps, layers, h = case["batch"], case["steps"], case["layers"], shape["hidden"]
    n_bytes = n_flops = 0
    for s in range(steps):
        kv_row = 2 * shape["n_kv_heads"] * shape["head_dim"]
        for _, M, K in _projections(shape):
            n_bytes += layers * M * blocks_per_row(K) * BLOCK_BYTES[kind]
            n_flops += layers * 2 * M * K * b
        n_bytes += layers * b * 4 * kv_row * (case["context"] + s + 1)
        n_flops += layers * b * 4 * shape["n_heads"] * shape["head_dim"] * (case["context"] + s + 1)
        n_bytes += b * blocks_per_row(h) * BLOCK_BYTES[INT8]
        # the head: every step leaves its logits on the device; to the host only where they are asked for
        n_bytes += case["vocab"] * blocks_per_row(h) * BLOCK_BYTES[INT8]
        n_bytes += 4 * b * case["vocab"] * (2 if case["logits"] == "every" or s + 1 == steps else 1)
        n_flops += 2 * case["vocab"] * h * b
    return {"bytes": n_bytes, "flops": n_flops}


def tolerance(case):
    if case["op"] == "quantize":
        # scales are fp32 sums or maxima of a block; a code next to a rounding tie may move with a scale's last bit
        return {"rel": 1e-6, "differ": 1e-5}
    if case["op"] == "decode":
        # fp32 sums in another order, carried through the layers: what two fp32 implementations of a step differ by
        return {"rel": 3e-5}
    return {"rel": 1e-5}


# ---- inputs ------------------------------------------------------------------------------------------------

class _Random:
    """Seeded draws on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE)
        self.g.manual_seed(int(seed))

    def bytes(self, *shape):
        return torch.randint(0, 256, shape, dtype=torch.uint8, device=DEVICE, generator=self.g)

    def uniform(self, lo, hi, *shape):
        return torch.rand(shape, device=DEVICE, generator=self.g) * (hi - lo) + lo

    def normal(self, *shape):
        return torch.randn(shape, device=DEVICE, generator=self.g)

    def tokens(self, n, vocab):
        return torch.randint(0, vocab, (n,), device=DEVICE, generator=self.g).cpu().numpy()

    def activations(self, n):
        """N(0,1) with 1 % of the positions ten times as large."""
        x = self.normal(n)
        return torch.where(self.uniform(0, 1, n) < 0.01, 10 * x, x).cpu().numpy()


def _real_bits(K):
    """[blocks, 32] bytes with the bits of the columns below K set, most significant bit first."""
    m = np.zeros(blocks_per_row(K) * 256, np.uint8)
    m[:K] = 1
    return torch.from_numpy(np.packbits(m).reshape(-1, 32)).to(DEVICE)


def _tensor(r, kind, M, K, lo=0.01, hi=0.05, name=""):
    """A weight matrix of the block kind: uniform codes (ternary: a third each), scales as a quantizer
    leaves them for weights of magnitude lo to hi, neutral codes in the padding columns."""
    bpr = blocks_per_row(K)
    row_scales = kind in (TERNARY, BINARY, INT2)
    s = r.uniform(lo, hi, M, 1 if row_scales else bpr).expand(M, bpr).contiguous()
    if kind == TERNARY:
        zero = r.bytes(M, bpr, 32)
        for step in (1, 0, 1, 0, 1, 0):  # bits of 1/3 from the last one up
            zero = (zero | r.bytes(M, bpr, 32)) if step else (zero & r.bytes(M, bpr, 32))
        zero = zero | ~_real_bits(K)
        parts = [r.bytes(M, bpr, 32) & ~zero, zero, s]
    elif kind == INT2:
        parts = [r.bytes(M, bpr, 64), s, s * r.uniform(0.2, 0.5, M, 1)]
    elif kind == INT8:
        d = r.bytes(M, bpr * 256)
        d[:, K:] = 0
        parts = [s / 127.0, torch.where(d == 128, d + 1, d).view(M, bpr, 256)]
    elif kind == INT4:
        codes = r.bytes(M, bpr * 128)
        if K % 256:
            codes[:, (K + 1) // 2:] = 0x88
            if K % 2:
                codes[:, K // 2] = codes[:, K // 2] & 0xF0 | 8
        parts = [codes.view(M, bpr, 128), s / 8.0]
    elif kind == BINARY:
        parts = [r.bytes(M, bpr, 32), s]
    else:
        parts = [r.bytes(M, bpr, 32 * kind), s / float(1 << (kind - 1))]
    raw = torch.cat([p.contiguous().view(M, bpr, -1).view(torch.uint8) if p.dtype == torch.uint8
                     else p.contiguous().view(M, bpr, 1).view(torch.uint8) for p in parts], dim=2)
    return PackedTensor(kind, raw.cpu().numpy().reshape(-1).view(BLOCK_DTYPES[kind]), M, K, DEFAULT_QUANT_BITS[kind], name)


class _View:
    """A device buffer of the library as an fp32 array for the CUDA array interface."""

    def __init__(self, buf, shape):
        self.buf = buf
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4", "data": (buf.ptr.value, False), "version": 3}


def _as_torch(buf, *shape):
    return torch.as_tensor(_View(buf, shape), device=DEVICE)


def prepare(case, seed):
    r = _Random(seed)
    return {"linear": _prepare_linear, "group": _prepare_group, "host": _prepare_host, "quantize": _prepare_quantize,
            "decode": _prepare_decode}[case["op"]](case, r)


def _prepare_linear(case, r):
    ctx = default_context()
    M, K, b = case["M"], case["K"], case["batch"]
    st = {"op": "linear", "ctx": ctx, "w": ctx.upload(_tensor(r, KINDS[case["kind"]], M, K)), "batch": b,
          "x": ctx.to_device(r.activations(b * K)), "y": ctx.malloc(4 * b * M),
          "bias": ctx.to_device(r.normal(M).cpu().numpy()) if case["bias"] else None}
    st["out"] = _as_torch(st["y"], b, M)
    return st


def _prepare_group(case, r):
    ctx = default_context()
    ws, xs, ys = [], [], []
    for _ in range(case["layers"]):
        for _, M, K in _projections(synth.MODEL_SHAPES[case["shape"]]):
            ws.append(ctx.upload(_tensor(r, KINDS[case["kind"]], M, K)))
            xs.append(ctx.to_device(r.activations(K)))
            ys.append(ctx.malloc(4 * M))
    return {"op": "group", "group": Group(ctx, ws, xs, ys), "out": [_as_torch(y, w.M) for w, y in zip(ws, ys)]}


def _prepare_host(case, r):
    t = _tensor(r, KINDS[case["kind"]], case["M"], case["K"])
    ctx = default_context()
    t._device = ctx.upload(t)  # lut_linear keeps the device copy with the tensor; a program makes it once
    return {"op": "host", "w": t, "batch": case["batch"], "x": r.activations(case["batch"] * case["K"]),
            "bias": r.normal(case["M"]).cpu().numpy() if case["bias"] else None}


def _prepare_quantize(case, r):
    return {"op": "quantize", "kind": KINDS[case["kind"]], "rotate": case["rotate"],
            "w": (0.02 * r.normal(case["M"], case["K"])).cpu().numpy()}


def _prepare_decode(case, r):
    shape = dict(synth.MODEL_SHAPES[case["shape"]], n_layers=case["layers"], vocab=case["vocab"], max_seq=MAX_SEQ)
    kind, h = KINDS[case["kind"]], shape["hidden"]
    embed = _tensor(r, INT8, case["vocab"], h, 0.5, 1.5, name="model.embed_tokens.weight")
    head = PackedTensor(INT8, embed.blocks, embed.M, embed.K, embed.quant_bits, "lm_head.weight")

    def vector(n, mean, spread):
        return (mean + spread * r.normal(n)).cpu().numpy()

    layers = []
    for _ in range(min(2, case["layers"])):  # two layers of values; every layer has device copies of its own
        layer = {name: _tensor(r, kind, M, K, name=name) for name, M, K in _projections(shape)}
        layer["input_norm"], layer["post_norm"] = vector(h, 1.0, 0.1), vector(h, 1.0, 0.1)
        if shape["qkv_bias"]:
            for name in ("q", "k", "v"):
                layer[name + "_bias"] = vector(layer[name].M, 0.0, 0.02)
        layers.append(layer)
    spec = synth.ModelSpec(shape, embed, head, vector(h, 1.0, 0.1), [layers[i % len(layers)] for i in range(case["layers"])])
    model = Model(spec, default_context(), max_batch=case["batch"])
    if case["context"]:
        host = torch.empty(case["layers"] * 2 * MAX_SEQ * shape["n_kv_heads"] * shape["head_dim"], pin_memory=True)
        for seq in range(case["batch"]):
            host.copy_(0.1 * r.normal(host.numel()))
            model.kv_import(host.numpy(), seq)
    feed = []
    for s in range(case["steps"]):
        tokens, position = r.tokens(case["batch"], case["vocab"]), case["context"] + s
        feed.append((int(tokens[0]), position) if case["batch"] == 1 else (tokens.astype(np.int32), [position] * case["batch"]))
    return {"op": "decode", "model": model, "feed": feed, "every": case["logits"] == "every"}


# ---- one pass ------------------------------------------------------------------------------------------------

def run(state):
    op = state["op"]
    if op == "linear":
        state["ctx"].linear(state["w"], state["x"], state["y"], batch=state["batch"], bias=state["bias"])
        return state["out"]
    if op == "group":
        state["group"].launch()
        return state["out"]
    if op == "host":
        return lut_linear(state["w"], state["bias"], state["x"], None, state["batch"])
    if op == "quantize":
        blocks = quantize_tensor(state["kind"], state["w"], state["rotate"]).blocks
        return {name: blocks[name] for name in blocks.dtype.names}
    model, feed, every = state["model"], state["feed"], state["every"]
    for token, position in feed[:-1]:  # their keys and values stay in the cache and enter the last logits
        model.forward(token, position, fetch=every)
    token, position = feed[-1]
    return model.forward(token, position)


# ---- the same in 64 bits -----------------------------------------------------------------------------------

def _unpack(raw, bits):
    """[..., bytes] of a most-significant-bit-first stream as [..., codes] of `bits` bits each."""
    planes = torch.stack([(raw >> (7 - i)) & 1 for i in range(8)], dim=-1).flatten(-2)
    codes = planes.unflatten(-1, (-1, bits)).double()
    return codes @ torch.tensor([float(1 << (bits - 1 - i)) for i in range(bits)], dtype=torch.float64, device=raw.device)


def _dense(t):
    """The weights of a tensor as fp64 [M, padded K]."""
    def part(name):
        a = np.ascontiguousarray(t.blocks[name])
        return torch.from_numpy(a.view(np.uint8) if a.dtype == np.int8 else a.copy()).to(DEVICE)

    s = part("scale").double()[:, None]
    if t.kind == TERNARY:
        w = (1 - _unpack(part("zero_plane"), 1)) * (1 - 2 * _unpack(part("sign_plane"), 1)) * s
    elif t.kind == BINARY:
        w = (2 * _unpack(part("data"), 1) - 1) * s
    elif t.kind == INT2:
        b = _unpack(part("data"), 1).unflatten(-1, (-1, 2))
        w = (2 * b[..., 0] - 1) * s + (2 * b[..., 1] - 1) * part("scale2").double()[:, None]
    elif t.kind == INT8:
        w = part("data").view(torch.int8).double() * s
    else:
        w = (_unpack(part("data"), t.kind) - float(1 << (t.kind - 1))) * s
    return w.view(t.M, -1)


def _linear_exact(t, x, batch, bias=None):
    xs = torch.zeros(batch, blocks_per_row(t.K) * 256, dtype=torch.float64, device=DEVICE)
    xs[:, :t.K] = torch.from_numpy(x).to(DEVICE).double().view(batch, t.K)
    if t.kind in (TERNARY, BINARY, INT2):  # these kinds meet inputs rotated by a 256-point Hadamard transform
        h = torch.ones(1, 1, dtype=torch.float64, device=DEVICE)
        for _ in range(8):
            h = torch.cat([torch.cat([h, h], 1), torch.cat([h, -h], 1)], 0)
        xs = (xs.view(-1, 256) @ h / 16).view(batch, -1)
    y = xs @ _dense(t).T
    return y if bias is None else y + torch.from_numpy(bias).to(DEVICE).double()


def exact(case, seed):
    """What run() returns in 64 bits, for the projections; the quantizers' and decode steps' own arithmetic has
    oracles in the tests."""
    r = _Random(seed)
    if case["op"] == "linear":
        t = _tensor(r, KINDS[case["kind"]], case["M"], case["K"])
        x = r.activations(case["batch"] * case["K"])
        return _linear_exact(t, x, case["batch"], r.normal(case["M"]).cpu().numpy() if case["bias"] else None)
    if case["op"] == "host":
        t = _tensor(r, KINDS[case["kind"]], case["M"], case["K"])
        x = r.activations(case["batch"] * case["K"])
        return _linear_exact(t, x, case["batch"], r.normal(case["M"]).cpu().numpy() if case["bias"] else None).flatten().cpu().numpy()
    if case["op"] == "group":
        out = []
        for _ in range(case["layers"]):
            for _, M, K in _projections(synth.MODEL_SHAPES[case["shape"]]):
                t = _tensor(r, KINDS[case["kind"]], M, K)
                out.append(_linear_exact(t, r.activations(K), 1).flatten())
        return out
    return None
