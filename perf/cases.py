"""The work a program gives this library, as cases that can be timed and compared.

Twelve kinds cover one language model served from quantised weights: converting its weights, bringing a prompt
in (short, long, with quantised activations), generating token by token (projection by projection, a few tokens
at once, or a whole decoder step), the two ends of a step (embedding lookup and vocabulary projection), decode
attention on its own, and weights with zero points.  Sizes are those of the benchmark and the tests of this
repository or generic ones.  Every kind has one listed case and a range that `draw` samples.

Activations are drawn from N(0, 1) and weights from N(0, 0.02), in the sliced layout [ceil(C/4)][tokens][4] that
the operator takes by default.
"""
import importlib
import math

import torch

mld = importlib.import_module("ml-drift_b200")

PRECISION = {"f32": mld.F32, "f16": mld.F16, "f32f16": mld.F32F16}


def listed():
    return [
        # The smallest operator call: one fp32 token through an INT8 per-channel projection with a bias.
        {"name": "gemv_int8_f32", "kind": "fc", "k": 2048, "n": 2048, "tokens": 1, "bits": 8, "block": 0,
         "precision": "f32", "zero_point": False, "bias": True, "act_quant": 0},
        # Decode, one token: the FFN up-projection in INT4 with a scale per 32 inputs.
        {"name": "gemv_int4", "kind": "fc", "k": 2048, "n": 16384, "tokens": 1, "bits": 4, "block": 32,
         "precision": "f32f16", "zero_point": False, "bias": False, "act_quant": 0},
        # A handful of tokens at once: a few sequences decoded together, or a drafted continuation being checked.
        {"name": "batch5_int4", "kind": "fc", "k": 4096, "n": 11008, "tokens": 5, "bits": 4, "block": 32,
         "precision": "f32f16", "zero_point": False, "bias": False, "act_quant": 0},
        # Token in, logits out: embedding lookup and vocabulary projection over one INT8 table.
        {"name": "vocabulary_int8", "kind": "vocabulary", "vocab": 151936, "dim": 2048, "tokens": 1, "bits": 8,
         "block": 0},
        # A chat turn's worth of prompt tokens, a ragged count.
        {"name": "prompt77_int4", "kind": "fc", "k": 4096, "n": 11008, "tokens": 77, "bits": 4, "block": 32,
         "precision": "f32f16", "zero_point": False, "bias": False, "act_quant": 0},
        # A long prompt: the weights arrive packed on every call, as in a graph with external weights.
        {"name": "prompt1024_int4", "kind": "fc", "k": 4096, "n": 14336, "tokens": 1024, "bits": 4, "block": 32,
         "precision": "f32f16", "zero_point": False, "bias": False, "act_quant": 0},
        # The largest operator call: long prompt, INT8 weights, activations quantised per token inside the call.
        {"name": "prompt2048_w8a8", "kind": "fc", "k": 8192, "n": 28672, "tokens": 2048, "bits": 8, "block": 0,
         "precision": "f32f16", "zero_point": False, "bias": False, "act_quant": 2},
        # One generated token of the 7B geometry at a cache of 2048 tokens: the headline workload.
        {"name": "decoder_7b", "kind": "decoder", "layers": 32, "heads": 32, "ffn": 11008, "max_seq": 2048,
         "pos": 2047, "block": 32, "host": False},
        # A small decoder early in a conversation, driven from host vectors as a token loop on the CPU does.
        {"name": "decoder_small_host", "kind": "decoder", "layers": 8, "heads": 8, "ffn": 2816, "max_seq": 512,
         "pos": 100, "block": 32, "host": True},
        # Decode attention alone over a long cache with a ragged length.
        {"name": "attention_8191", "kind": "attention", "heads": 32, "tokens": 8191},
        # Loading a checkpoint: fp32 projection -> INT4 values and scales -> the operator's layouts.
        {"name": "convert_int4", "kind": "convert", "k": 4096, "n": 14336, "bits": 4, "block": 32},
        # Asymmetrically quantised weights (a zero point per scale), a short prompt.
        {"name": "zero_point_int4", "kind": "fc", "k": 2048, "n": 4096, "tokens": 12, "bits": 4, "block": 32,
         "precision": "f32f16", "zero_point": True, "bias": False, "act_quant": 0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi + 0.999)))


def _size(rng, lo, hi, multiple):
    """A size between lo and hi, spread over its logarithm, as a multiple of `multiple`."""
    return max(multiple, int(_log(rng, lo, hi)) // multiple * multiple)


def _fc(rng, k, n, tokens, bits, block, precision="f32f16", zero_point=False, act_quant=0):
    return {"kind": "fc", "k": k, "n": n, "tokens": tokens, "bits": bits, "block": block, "precision": precision,
            "zero_point": zero_point, "bias": rng.random() < 0.3, "act_quant": act_quant}


def _bits_block(rng):
    """INT4 with block scales (mostly 32 inputs) or per channel, INT8 per channel."""
    return rng.choice(((4, 32), (4, 32), (4, 64), (4, 128), (4, 0), (8, 0), (8, 0)))


def draw(rng):
    kind = rng.choice(("small", "gemv", "batch", "vocabulary", "short", "long", "w8a8", "decoder", "decoder_host",
                       "attention", "convert", "zero_point"))
    edge = rng.choice((64, 64, 8, 1))  # most projections are whole tiles, some are not
    if kind == "small":
        bits, block = rng.choice(((8, 0), (8, 0), (4, 32)))
        return _fc(rng, _size(rng, 256, 4096, 32 if block else rng.choice((64, 4, 1))), _size(rng, 256, 4096, edge), 1,
                   bits, block, precision="f32")
    if kind in ("gemv", "batch", "short"):
        bits, block = _bits_block(rng)
        k, n = _size(rng, 512, 14336, 128), _size(rng, 512, 28672, edge)
        if kind == "gemv":
            return _fc(rng, k, n, 1, bits, block, rng.choice(("f32f16", "f32f16", "f16")))
        if kind == "batch":
            precision = rng.choice(("f32f16", "f16"))
            return _fc(rng, k, n, rng.randint(2, 16 if precision == "f16" else 8), bits, block, precision)
        return _fc(rng, k, n, int(_log(rng, 9, 512)), bits, block)
    if kind == "vocabulary":
        bits, block = rng.choice(((8, 0), (8, 0), (4, 32)))
        return {"kind": "vocabulary", "vocab": _size(rng, 32000, 262144, rng.choice((64, 8))),
                "dim": _size(rng, 640, 2560, 128), "tokens": 1, "bits": bits, "block": block}
    if kind == "long":
        bits, block = _bits_block(rng)
        return _fc(rng, _size(rng, 1024, 8192, 128), _size(rng, 1024, 14336, rng.choice((64, 8))),
                   int(_log(rng, 513, 4096)), bits, block)
    if kind == "w8a8":
        return _fc(rng, _size(rng, 1024, 8192, 64), _size(rng, 1024, 14336, rng.choice((64, 8))),
                   int(_log(rng, 17, 4096)), 8, 0, act_quant=rng.choice((1, 2)))
    if kind in ("decoder", "decoder_host"):
        host = kind == "decoder_host"
        heads = int(_log(rng, 4, 16 if host else 32))
        max_seq = _size(rng, 64, 2048, 16)
        return {"kind": "decoder", "layers": int(_log(rng, 2, 12 if host else 24)), "heads": heads,
                "ffn": max(256, int(heads * 128 * rng.uniform(2.0, 3.0)) // 256 * 256), "max_seq": max_seq,
                "pos": rng.randrange(max_seq), "block": rng.choice((32, 32, 64, 128)), "host": host}
    if kind == "attention":
        return {"kind": "attention", "heads": rng.choice((8, 12, 16, 24, 32, 40)), "tokens": int(_log(rng, 16, 16384))}
    if kind == "convert":
        bits, block = _bits_block(rng)
        return {"kind": "convert", "k": _size(rng, 512, 11008, 128), "n": _size(rng, 512, 14336, edge), "bits": bits,
                "block": block}
    bits, block = rng.choice(((4, 32), (4, 128), (8, 0)))
    return _fc(rng, _size(rng, 512, 4096, 128), _size(rng, 512, 8192, edge), int(_log(rng, 1, 64)), bits, block,
               zero_point=True)


# ------------------------------------------------------------------ what a program has in hand before the call
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(gen, *shape):
    return torch.randn(shape, generator=gen, device="cuda")


def _activations(gen, channels, tokens, dtype):
    """[ceil(channels / 4)][tokens][4] with zeros in the padded channels."""
    slices = -(-channels // 4)
    x = _randn(gen, slices, tokens, 4)
    if channels % 4:
        x[-1, :, channels % 4:] = 0
    return x.to(dtype)


def _symmetric(gen, n, k, bits, block, f16=True, want_sum=False):
    """Packed weights, scales (and input sums) of an N(0, 0.02) projection."""
    q, s = mld.quantize_weights(_randn(gen, n, k).mul_(0.02), bits, block)
    packed, sums = mld.pack_weights(q, (n, 1, 1, k), bits, want_sum=want_sum)
    return packed, mld.pack_scales(s, f16), sums


def _asymmetric(gen, n, k, bits, block, f16=True):
    """Packed weights, scales and zero points: w = (q - zero_point) * scale over each group's own range."""
    w = _randn(gen, n, k).mul_(0.02).reshape(n, -1, block or k)
    low, high = w.amin(-1, keepdim=True), w.amax(-1, keepdim=True)
    top, offset = 2 ** bits - 1, 2 ** (bits - 1)
    scale = (high - low) / top
    zero = torch.round(-low / scale) - offset
    q = torch.clamp(torch.round(w / scale) + zero, -offset, offset - 1).to(torch.int8).reshape(n, k)
    packed, _ = mld.pack_weights(q, (n, 1, 1, k), bits)
    return packed, mld.pack_scales(scale[..., 0], f16), mld.pack_scales(zero[..., 0], f16)


def _prepare_fc(c, gen):
    f16 = c["precision"] != "f32"
    n, k, tokens = c["n"], c["k"], c["tokens"]
    dtype = torch.float16 if f16 else torch.float32
    plan = mld.FullyConnectedPlan(
        n, k, c["bits"], scale_mode=mld.SCALE_BLOCK if c["block"] else mld.SCALE_PER_CHANNEL,
        groups=k // c["block"] if c["block"] else 1, has_zero_point=c["zero_point"], has_bias=c["bias"],
        precision=PRECISION[c["precision"]], max_tokens=tokens, prefill_act_quant=c["act_quant"])
    zero = None
    if c["zero_point"]:
        packed, scale, zero = _asymmetric(gen, n, k, c["bits"], c["block"], f16)
    else:
        packed, scale, sums = _symmetric(gen, n, k, c["bits"], c["block"], f16, want_sum=c["act_quant"] == 2)
        if c["act_quant"] == 2:
            plan.set_weights_sum(sums)
    slices = -(-n // 4)
    bias = None
    if c["bias"]:
        bias = torch.zeros(slices * 4, dtype=dtype, device="cuda")
        bias[:n] = _randn(gen, n).mul_(0.01).to(dtype)
    return {"plan": plan, "x": _activations(gen, k, tokens, dtype), "weights": packed, "scale": scale, "zero": zero,
            "bias": bias, "y": torch.empty((slices, tokens, 4), dtype=dtype, device="cuda"), "tokens": tokens}


def _prepare_vocabulary(c, gen):
    vocab, dim, block = c["vocab"], c["dim"], c["block"]
    mode, groups = (mld.SCALE_BLOCK, dim // block) if block else (mld.SCALE_PER_CHANNEL, 1)
    packed, scale, _ = _symmetric(gen, vocab, dim, c["bits"], block)
    return {"plan": mld.FullyConnectedPlan(vocab, dim, c["bits"], scale_mode=mode, groups=groups, max_tokens=1),
            "ids": torch.randint(0, vocab, (c["tokens"],), generator=gen, device="cuda", dtype=torch.int32),
            "hidden": _activations(gen, dim, 1, torch.float16), "weights": packed, "scale": scale, "mode": mode,
            "groups": groups, "vocab": vocab, "dim": dim, "bits": c["bits"],
            "x": torch.empty((c["tokens"], dim), dtype=torch.float16, device="cuda"),
            "logits": torch.empty((-(-vocab // 4), 1, 4), dtype=torch.float16, device="cuda")}


def _prepare_decoder(c, gen):
    heads, ffn, layers, block = c["heads"], c["ffn"], c["layers"], c["block"]
    d = heads * 128
    decoder = mld.Decoder(layers, d, heads, ffn, c["max_seq"], block=block)
    k_cache = _randn(gen, layers, c["max_seq"], d).half()
    v_cache = _randn(gen, layers, c["max_seq"], d).half()
    for layer in range(layers):
        tensors = {}
        for name, n, k in (("qkv", 3 * d, d), ("o", d, d), ("gu", 2 * ffn, d), ("down", d, ffn)):
            tensors["w" + name], tensors["s" + name], _ = _symmetric(gen, n, k, 4, block)
        for name in ("norm1", "norm2"):
            tensors[name] = (1.0 + 0.1 * _randn(gen, d)).half()
        decoder.set_layer(layer, kcache=k_cache[layer], vcache=v_cache[layer], **tensors)
    x = _randn(gen, d).half()
    y = torch.empty_like(x)
    if c["host"]:
        x, y = x.cpu().pin_memory(), torch.empty(d, dtype=torch.float16).pin_memory()
    return {"decoder": decoder, "x": x, "y": y, "k_cache": k_cache, "v_cache": v_cache, "pos": c["pos"],
            "host": c["host"]}


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "fc":
        state = _prepare_fc(case, gen)
    elif kind == "vocabulary":
        state = _prepare_vocabulary(case, gen)
    elif kind == "decoder":
        state = _prepare_decoder(case, gen)
    elif kind == "attention":
        heads, tokens = case["heads"], case["tokens"]
        state = {"q": (_randn(gen, heads, 128) / math.sqrt(128)).half(), "k": _randn(gen, tokens, heads * 128).half(),
                 "v": _randn(gen, tokens, heads * 128).half(), "heads": heads, "tokens": tokens,
                 "out": torch.empty((heads, 128), dtype=torch.float16, device="cuda")}
    else:
        state = {"w": _randn(gen, case["n"], case["k"]).mul_(0.02), "bits": case["bits"], "block": case["block"]}
    state["kind"] = kind
    return state


# ------------------------------------------------------------------------------------------------- one pass
def run(state):
    kind, s = state["kind"], state
    if kind == "fc":
        s["plan"].run(s["x"], s["weights"], s["scale"], s["y"], s["tokens"], zero_point=s["zero"], bias=s["bias"])
        return s["y"]
    if kind == "vocabulary":
        mld.embedding_lookup(s["ids"], s["weights"], s["scale"], s["x"], s["vocab"], s["dim"], s["bits"],
                             scale_mode=s["mode"], groups=s["groups"])
        s["plan"].run(s["hidden"], s["weights"], s["scale"], s["logits"], 1)
        return s["x"], s["logits"]
    if kind == "decoder":
        step = s["decoder"].step_host if s["host"] else s["decoder"].step
        step(s["x"], s["y"], s["pos"])
        return s["y"], s["k_cache"], s["v_cache"]
    if kind == "attention":
        mld.attn_decode(s["q"], s["k"], s["v"], s["out"], s["heads"], s["tokens"])
        return s["out"]
    q, scale = mld.quantize_weights(s["w"], s["bits"], s["block"])
    packed, sums = mld.pack_weights(q, (q.shape[0], 1, 1, q.shape[1]), s["bits"], want_sum=True)
    return packed, mld.pack_scales(scale, True), sums


# ------------------------------------------------------------------------ the same in 64 bits, by plain torch
def _over(a, b):
    """a / b, rounded once (with a plain number on either side torch multiplies by a reciprocal instead)"""
    return torch.div(*(t if torch.is_tensor(t) else torch.tensor(t, device="cuda") for t in (a, b)))


def _quantised(w, bits, block):
    """(integers, scales [n][groups]): the largest magnitude of a row or block maps to 127 (7), halves round to even."""
    n, k = w.shape
    blocks = w.reshape(n, -1, block if bits == 4 and block else k)
    top = 127.0 if bits == 8 else 7.0
    scale = _over(blocks.abs().amax(-1), top)
    scale = torch.where(scale == 0, torch.ones_like(scale), scale)
    return torch.round(blocks / scale[..., None]).clamp_(-top - 1, top).to(torch.int8), scale


def _weights64(gen, n, k, bits, block, dtype, zero_point=False):
    """The [n][k] weights that the packed tensors stand for, drawn as _symmetric and _asymmetric draw them."""
    w = _randn(gen, n, k).mul_(0.02)
    if not zero_point:
        q, scale = _quantised(w, bits, block)
        return (q.double() * scale.to(dtype).double()[..., None]).reshape(n, k)
    w = w.reshape(n, -1, block or k)
    low, high = w.amin(-1, keepdim=True), w.amax(-1, keepdim=True)
    top, offset = 2 ** bits - 1, 2 ** (bits - 1)
    scale = (high - low) / top
    zero = torch.round(-low / scale) - offset
    q = torch.clamp(torch.round(w / scale) + zero, -offset, offset - 1)
    return ((q.double() - zero.to(dtype).double()) * scale.to(dtype).double()).reshape(n, k)


def _rows(x, channels):
    """[slices][tokens][4] -> [tokens][channels]"""
    return x.permute(1, 0, 2).reshape(x.shape[1], -1)[:, :channels]


def _sliced(y):
    """[tokens][channels] -> [slices][tokens][4], zeros in the padded channels"""
    y = torch.nn.functional.pad(y, (0, -y.shape[1] % 4))
    return y.reshape(y.shape[0], -1, 4).permute(1, 0, 2).contiguous()


def _act_quantised(x, symmetric):
    """The value that each activation stands for after its quantisation to 8 bits per token (a 32-bit rule)."""
    x = x.float()
    if symmetric:
        inv = torch.clamp(_over(x.abs().amax(1, keepdim=True), 127.0), min=2.0 ** -14)
        q = torch.floor(x * _over(1.0, inv) + 128.5).clamp(0, 255) - 128
        return q.double() * inv.double()
    low, high = x.amin(1, keepdim=True), x.amax(1, keepdim=True)
    span = high - low
    q = ((x - low) * _over(255.0, span) + 0.5).to(torch.int32).clamp(0, 255) - 128
    return q.double() * _over(span, 255.0).double() + (low + span * (128.0 / 255.0)).double()


def _exact_fc(c, gen):
    dtype = torch.float32 if c["precision"] == "f32" else torch.float16
    w = _weights64(gen, c["n"], c["k"], c["bits"], c["block"], dtype, c["zero_point"])
    bias = _randn(gen, c["n"]).mul_(0.01).to(dtype).double() if c["bias"] else 0.0
    x = _rows(_activations(gen, c["k"], c["tokens"], dtype), c["k"])
    x = _act_quantised(x, c["act_quant"] == 1) if c["act_quant"] and c["tokens"] > 8 else x.double()
    return _sliced(x @ w.T + bias)


def _rope64(v, pos):
    half = v.shape[-1] // 2
    angle = pos / 1.0e6 ** (torch.arange(half, dtype=torch.float64, device=v.device) / half)
    c, s, a, b = torch.cos(angle), torch.sin(angle), v[..., :half], v[..., half:]
    return torch.cat((a * c - b * s, b * c + a * s), -1)


def _attend64(q, k, v):
    """q [heads][128], k and v [tokens][heads][128]"""
    return torch.einsum("ht,thd->hd", torch.softmax(torch.einsum("hd,thd->ht", q, k), 1), v)


def _exact_decoder(c, gen):
    heads, ffn, layers, pos = c["heads"], c["ffn"], c["layers"], c["pos"]
    d = heads * 128
    k_cache = _randn(gen, layers, c["max_seq"], d).half().double()
    v_cache = _randn(gen, layers, c["max_seq"], d).half().double()
    stack = []
    for _ in range(layers):
        weights = [_quantised(_randn(gen, n, k).mul_(0.02), 4, c["block"])
                   for n, k in ((3 * d, d), (d, d), (2 * ffn, d), (d, ffn))]
        stack.append((weights, [(1.0 + 0.1 * _randn(gen, d)).half().double() for _ in range(2)]))
    x = _randn(gen, d).half().double()

    def project(weight, v):
        q, scale = weight
        return (q.double() * scale.half().double()[..., None]).reshape(q.shape[0], -1) @ v

    def norm(v, gamma):
        return v * torch.rsqrt(v.square().mean() + 1e-6) * gamma

    for layer, ((qkv, o, gate_up, down), (gamma1, gamma2)) in enumerate(stack):
        q, k, v = project(qkv, norm(x, gamma1)).reshape(3, heads, 128)
        k_cache[layer, pos], v_cache[layer, pos] = _rope64(k, pos).reshape(-1), v.reshape(-1)
        keys, values = (t[layer, :pos + 1].reshape(pos + 1, heads, 128) for t in (k_cache, v_cache))
        x = x + project(o, _attend64(_rope64(q, pos) / math.sqrt(128), keys, values).reshape(-1))
        gate, up = project(gate_up, norm(x, gamma2)).reshape(ffn, 2).T  # rows alternate gate, up
        x = x + project(down, torch.nn.functional.silu(gate) * up)
    return (x.cpu() if c["host"] else x), k_cache, v_cache


def exact(case, seed):
    gen = _generator(seed)
    c, kind = case, case["kind"]
    if kind == "fc":
        return _exact_fc(c, gen)
    if kind == "vocabulary":
        w = _weights64(gen, c["vocab"], c["dim"], c["bits"], c["block"], torch.float16)
        ids = torch.randint(0, c["vocab"], (c["tokens"],), generator=gen, device="cuda", dtype=torch.int32)
        hidden = _rows(_activations(gen, c["dim"], 1, torch.float16), c["dim"]).double()
        return w[ids.long()], _sliced(hidden @ w.T)
    if kind == "decoder":
        return _exact_decoder(c, gen)
    if kind == "attention":
        q = (_randn(gen, c["heads"], 128) / math.sqrt(128)).half().double()
        k, v = (_randn(gen, c["tokens"], c["heads"], 128).half().double() for _ in range(2))
        return _attend64(q, k, v)
    w = _randn(gen, c["n"], c["k"]).mul_(0.02).double()
    bound = w.reshape(c["n"], -1, c["block"] if c["bits"] == 4 and c["block"] else c["k"]).abs().amax(-1)
    scale = torch.nn.functional.pad(bound / (127.0 if c["bits"] == 8 else 7.0), (0, 0, 0, -c["n"] % 4))
    return None, scale.T.contiguous(), None  # (the other two are whole numbers)


# --------------------------------------------------------------------------- what a pass cannot do without
def _weights_bytes(n, k, bits, block, element, zero_point=False):
    n4, k4 = -(-n // 4) * 4, -(-k // 4) * 4
    return n4 * k4 * bits // 8 + n4 * (k // block if block else 1) * element * (2 if zero_point else 1)


def work(case):
    c, kind = case, case["kind"]
    if kind == "fc":
        element = 4 if c["precision"] == "f32" else 2
        weights = _weights_bytes(c["n"], c["k"], c["bits"], c["block"], element, c["zero_point"])
        vectors = (c["k"] * c["tokens"] + c["n"] * (c["tokens"] + (1 if c["bias"] else 0))) * element
        return {"bytes": weights + vectors, "flops": 2.0 * c["tokens"] * c["n"] * c["k"]}
    if kind == "vocabulary":
        vectors = (c["dim"] * (1 + c["tokens"]) + c["vocab"]) * 2
        row = c["tokens"] * c["dim"] * c["bits"] // 8
        return {"bytes": _weights_bytes(c["vocab"], c["dim"], c["bits"], c["block"], 2) + vectors + row,
                "flops": 2.0 * c["vocab"] * c["dim"]}
    if kind == "decoder":
        d, ffn = c["heads"] * 128, c["ffn"]
        weights = sum(_weights_bytes(n, k, 4, c["block"], 2) for n, k in ((3 * d, d), (d, d), (2 * ffn, d), (d, ffn)))
        cache = 2 * (c["pos"] + 1) * d * 2
        values = 4 * d * d + 3 * d * ffn
        return {"bytes": c["layers"] * (weights + cache + 4 * d) + 4 * d,
                "flops": c["layers"] * (2.0 * values + 4.0 * (c["pos"] + 1) * d)}
    if kind == "attention":
        width = c["heads"] * 128
        return {"bytes": 2 * c["tokens"] * width * 2 + 2 * width * 2, "flops": 4.0 * c["tokens"] * width}
    return {"bytes": c["n"] * c["k"] * 4 + _weights_bytes(c["n"], c["k"], c["bits"], c["block"], 2) + c["n"] * 4,
            "flops": 2.0 * c["n"] * c["k"]}


# ------------------------------------------------------------- how far another correct implementation may be off
#
# Measured against the same product in fp64 (2-norm of the difference over 2-norm), stated about four times over:
#   fp32 tensors                          1.6e-7  (a single running fp32 sum over K = 4096 shows up to 1e-6)
#   fp16 tensors, fp32 sums               2.1e-4  (the rounding of the result)
#   the same, weights dequantised to fp16 3.6e-4
#   the same, products summed in half     5.8e-4  (the general decode kernel)
#   int8 activations                      2.1e-4  beyond the quantisation itself, whose integers are exact
#   attention                             2.1e-4
# Decoder: the same steps as one kernel and as a chain of operators, which add and round in different places;
# the difference grows with the layers it passes (2 layers 4.7e-4, 6: 1.4e-3, 15: 3.3e-3, 32: 4.4e-3).
def tolerance(case):
    kind = case["kind"]
    if kind == "convert":
        return "exact"
    if kind == "decoder":
        rel = min(1.75e-2, 2e-3 + 7e-4 * case["layers"])
        return {"rel": rel, "max": 4 * rel}
    if kind == "fc" and case["precision"] == "f32":
        return {"rel": 1e-6, "max": 4e-6}
    if kind == "fc" and not case["act_quant"]:
        rel = 2e-3 if case["zero_point"] or case["n"] % 8 else 1.5e-3
        return {"rel": rel, "max": 5 * rel}
    return {"rel": 1e-3, "max": 5e-3}
