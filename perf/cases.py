"""The work a program has the framework do, as cases that can be timed and whose outputs can be compared.

Three kinds of case, each through the Python binding of the C ABI (`runtime`, `qmm`):

  mul_mat    activations [M][K] x quantized weight [N][K]^T through `qmm.MulMat`: one-shot (`run`: record, submit, wait, what
             a program with a single product does) or recorded once and replayed (what a token loop does)
  layer      one decoder layer on M new positions over a KV cache, recorded once and replayed: RMS norm, q / k / v, ROPE,
             cache update, attention, o + residual, RMS norm, gate / up, SWIGLU, down + residual, every op the way the
             binding offers it for that type and M (grouped launches and fused consumers for one row)
  attention  `ameva_flash_attn` alone on a long cache, recorded once and replayed

Weights are ggml blocks whose codes are normally distributed, as quantizers leave them; activations, caches and queries
are standard normal.
"""
import importlib
import math
import struct

import torch

amv = importlib.import_module("ameva-compute_b200")
rt, qmm = amv.runtime, amv.qmm

#: ggml type: (id, weights per block, bytes per block)
TYPES = {"q4_0": (2, 32, 18), "q5_0": (6, 32, 22), "q8_0": (8, 32, 34), "q4_K": (12, 256, 144), "q5_K": (13, 256, 176),
         "q6_K": (14, 256, 210), "i2_s": (36, 128, 32)}


def listed():
    return [
        # the smallest call: one product of one row, launched and waited for (4096 x 4096 is an attention projection)
        {"name": "call_q4_0_4096x4096_m1", "kind": "mul_mat", "type": "q4_0", "M": 1, "N": 4096, "K": 4096, "replay": False},
        # token generation, 7B-sized layer; v and down in Q6_K as in mixed Q4_K / Q6_K model files
        {"name": "layer_q4_K_4096_m1", "kind": "layer", "type": "q4_K", "alt": "q6_K", "M": 1, "heads": 32, "kv_heads": 32,
         "D": 128, "ff": 11008, "n_kv": 2048},
        # token generation, a small model whose width (896) is no multiple of 256: bound by launches and latency
        {"name": "layer_q8_0_896_m1", "kind": "layer", "type": "q8_0", "alt": "q8_0", "M": 1, "heads": 14, "kv_heads": 2,
         "D": 64, "ff": 4864, "n_kv": 333},
        # token generation, ternary 2B-sized layer
        {"name": "layer_i2_s_2560_m1", "kind": "layer", "type": "i2_s", "alt": "i2_s", "M": 1, "heads": 20, "kv_heads": 5,
         "D": 128, "ff": 6912, "n_kv": 777},
        # a prompt's last chunk of 512 positions, 8B-sized layer with grouped KV heads
        {"name": "layer_q4_0_4096_m512", "kind": "layer", "type": "q4_0", "alt": "q4_0", "M": 512, "heads": 32, "kv_heads": 8,
         "D": 128, "ff": 14336, "n_kv": 2048},
        # a few sequences or drafted tokens at once
        {"name": "q4_K_11008x4096_m8", "kind": "mul_mat", "type": "q4_K", "M": 8, "N": 11008, "K": 4096, "replay": True},
        # token generation, projection of a 70B-sized layer
        {"name": "q4_K_28672x8192_m1", "kind": "mul_mat", "type": "q4_K", "M": 1, "N": 28672, "K": 8192, "replay": True},
        # the prompt product the benchmark's headline is quoted on
        {"name": "q8_0_11008x4096_m512", "kind": "mul_mat", "type": "q8_0", "M": 512, "N": 11008, "K": 4096, "replay": True},
        # a short prompt of odd length on a weight with an odd number of rows
        {"name": "q5_K_3203x3328_m77", "kind": "mul_mat", "type": "q5_K", "M": 77, "N": 3203, "K": 3328, "replay": True},
        # a prompt on ternary weights
        {"name": "i2_s_6912x2560_m128", "kind": "mul_mat", "type": "i2_s", "M": 128, "N": 6912, "K": 2560, "replay": True},
        # the largest: a long prompt on a 70B-sized projection
        {"name": "q4_K_28672x8192_m2048", "kind": "mul_mat", "type": "q4_K", "M": 2048, "N": 28672, "K": 8192, "replay": True},
        # token generation at a long context
        {"name": "attention_1x32768", "kind": "attention", "heads": 32, "kv_heads": 8, "D": 128, "n_q": 1, "n_kv": 32768},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _heads(rng, width, widest):
    """heads, kv_heads, D: a layer's width is a multiple of `width` and at most `widest`."""
    D = rng.choice([64, 128, 128])
    while True:
        kv_heads, group = rng.randint(1, 32), rng.randint(1, 8)
        if kv_heads * group * D % width == 0 and kv_heads * group * D <= widest:
            return kv_heads * group, kv_heads, D


def draw(rng):
    kind = rng.choice(["mul_mat"] * 6 + ["layer"] * 3 + ["attention"])
    if kind == "mul_mat":
        t = rng.choice(["q4_0", "q5_0", "q8_0", "q4_K", "q4_K", "q5_K", "q6_K", "i2_s"])
        M = rng.choice([1, rng.randint(2, 8), _log(rng, 9, 2048), _log(rng, 9, 2048)])
        if t in ("q4_0", "q5_0", "q8_0") and rng.random() < 0.2:   # widths that are no multiple of 256: small models
            M, N, K = min(M, 512), 2 * _log(rng, 128, 4096), 64 * rng.randint(9, 80)
        else:
            N, K = _log(rng, 256, 28672), 256 * _log(rng, 2, 112)
            N = min(N, 28672 * 8192 // K)
        return {"kind": kind, "type": t, "M": M, "N": N, "K": K, "replay": M > 1 or rng.random() < 0.5}
    if kind == "layer":
        t = rng.choice(["q4_0", "q8_0", "q4_K", "i2_s"])
        heads, kv_heads, D = _heads(rng, {"q4_K": 256, "i2_s": 128}.get(t, 64), 4096)
        M = rng.choice([1, 1, _log(rng, 2, 1024)])
        d = heads * D
        return {"kind": kind, "type": t, "alt": "q6_K" if t == "q4_K" else t, "M": M, "heads": heads, "kv_heads": kv_heads,
                "D": D, "ff": max(256, int(d * rng.uniform(2.5, 4.0)) // 256 * 256), "n_kv": max(M, _log(rng, 32, 8192))}
    heads, kv_heads, D = _heads(rng, 64, 8192)
    n_q = rng.choice([1, _log(rng, 2, 2048)])
    n_kv = min(_log(rng, 256, 32768), (1 << 37) // (n_q * heads * D))
    return {"kind": kind, "heads": heads, "kv_heads": kv_heads, "D": D, "n_q": n_q, "n_kv": max(n_q, n_kv)}


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def _products(c):
    """(type, N, K) of every weight of a case."""
    if c["kind"] == "mul_mat":
        return [(c["type"], c["N"], c["K"])]
    if c["kind"] == "attention":
        return []
    d, kv, ff, t, alt = c["heads"] * c["D"], c["kv_heads"] * c["D"], c["ff"], c["type"], c["alt"]
    return [(t, d, d), (t, kv, d), (alt, kv, d), (t, d, d), (t, ff, d), (t, ff, d), (alt, d, ff)]


def work(case):
    nbytes, flops = 0, 0
    M = case["M"] if "M" in case else case["n_q"]
    for t, N, K in _products(case):
        _, blk, blk_bytes = TYPES[t]
        nbytes += N * K // blk * blk_bytes
        flops += 2 * M * N * K
    if case["kind"] == "mul_mat":
        nbytes += 4 * M * (case["N"] + case["K"])
    else:
        d, n_kv = case["heads"] * case["D"], case["n_kv"]
        pairs = M * n_kv - M * (M - 1) // 2            # unmasked (position, key) pairs
        nbytes += 2 * n_kv * case["kv_heads"] * case["D"] * 2 + 2 * M * d * 4
        flops += 4 * pairs * d
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the path differs by from itself with exact integer products, from 64-bit sums (attention), or with
    its attention sums in another order (layers)."""
    if case["kind"] == "attention":
        return {"rel": 1e-3, "max": 0.04}     # queries and probabilities rounded to fp16: 2.6e-4, 9.6e-3 from 64-bit sums
    if case["kind"] == "layer":
        # 5.4e-3, 2.7e-2: attention and products as here, then rounded to 8 bits twice more, where a value near a tie moves by a
        # whole step
        return {"rel": 2e-2, "max": 0.12}
    if case["type"] == "i2_s" or case["M"] <= 8:
        return {"rel": 1e-5, "max": 1e-4}     # exact integers per block, summed in fp32
    return {"rel": 1.2e-3, "max": 8e-3}       # weights and activations rounded to fp16 once, summed in fp32: 3e-4, 2e-3


# ---- weights -----------------------------------------------------------------------------------------------------------
def _half_bytes(v):
    return v.to(torch.float16).view(-1, 1).view(torch.uint8)


def _nibbles(codes):
    """[n][64 c]: per 64 codes, 32 bytes with codes l and l + 32 (ggml's K-quant order)."""
    c = codes.view(codes.shape[0], -1, 2, 32)
    return (c[:, :, 0] | (c[:, :, 1] << 4)).reshape(codes.shape[0], -1)


def _six_bit(a, b):
    """Eight 6-bit scales and eight 6-bit minima in 12 bytes (Q4_K, Q5_K)."""
    return torch.cat([a[:, :4] | ((a[:, 4:] >> 4) << 6), b[:, :4] | ((b[:, 4:] >> 4) << 6), (a[:, 4:] & 15) | ((b[:, 4:] & 15) << 4)], 1)


def _ggml_blocks(t, N, K, std, gen):
    """ggml blocks of an [N][K] weight of standard deviation `std`, as host bytes."""
    _, blk, blk_bytes = TYPES[t]
    n = N * K // blk
    dev = gen.device

    def codes(mean, sigma, lo, hi, width=blk):
        v = torch.empty((n, width), device=dev).normal_(mean, sigma, generator=gen)
        return v.round_().clamp_(lo, hi).to(torch.int16)

    def about(v):      # block scales: positive, a fifth of spread
        return v * torch.empty(n, device=dev).normal_(1.0, 0.2, generator=gen).clamp_(0.4, 1.6)

    if t == "i2_s":    # two bits per weight: -1, 0, 1 as 0, 1, 2
        c = torch.randint(0, 3, (n, 4, 32), device=dev, dtype=torch.uint8, generator=gen)
        return (c[:, 0] << 6 | c[:, 1] << 4 | c[:, 2] << 2 | c[:, 3]).reshape(-1).cpu().numpy()
    u8 = torch.uint8
    if t == "q8_0":
        parts = [_half_bytes(about(std / 42.0)), codes(0, 42, -127, 127).to(torch.int8).view(u8)]
    elif t == "q4_0":
        q = codes(8, 2.9, 0, 15).to(u8)
        parts = [_half_bytes(about(std / 2.9)), q[:, :16] | (q[:, 16:] << 4)]
    elif t == "q5_0":
        q = codes(16, 5.8, 0, 31).to(u8)
        bits = (q >> 4).view(n, 4, 8) << torch.arange(8, device=dev, dtype=u8)
        parts = [_half_bytes(about(std / 5.8)), bits.sum(2, dtype=u8), (q[:, :16] & 15) | ((q[:, 16:] & 15) << 4)]
    elif t in ("q4_K", "q5_K"):
        top = 15 if t == "q4_K" else 31
        q = codes(top / 2, top / 5.2, 0, top).to(u8)
        six = _six_bit(codes(44, 9, 1, 63, 8).to(u8), codes(44, 9, 1, 63, 8).to(u8))
        d = about(std / (top / 5.2) / 44)
        parts = [_half_bytes(d), _half_bytes(d * (top / 2)), six]
        if t == "q5_K":    # bit of value e: byte e % 32, bit e / 32
            parts.append(((q >> 4).view(n, 8, 32) << torch.arange(8, device=dev, dtype=u8).view(1, 8, 1)).sum(1, dtype=u8))
        parts.append(_nibbles(q & 15))
    else:              # q6_K
        q = codes(32, 10, 0, 63).to(u8).view(n, 2, 4, 32)
        low = torch.cat([(q[:, :, 0] & 15) | ((q[:, :, 2] & 15) << 4), (q[:, :, 1] & 15) | ((q[:, :, 3] & 15) << 4)], 2)
        high = (q[:, :, 0] >> 4) | ((q[:, :, 1] >> 4) << 2) | ((q[:, :, 2] >> 4) << 4) | ((q[:, :, 3] >> 4) << 6)
        scales = codes(0, 60, -127, 127, 16).to(torch.int8).view(u8)
        parts = [low.reshape(n, 128), high.reshape(n, 64), scales, _half_bytes(about(std / 10 / 60))]
    return torch.cat(parts, 1).reshape(-1).cpu().numpy()


# ---- states ------------------------------------------------------------------------------------------------------------
_context = None


def _ctx():
    """A program has one context."""
    global _context
    if _context is None:
        _context = rt.init()
    return _context


class _State:
    """What the program holds between passes; everything it created is destroyed with it."""

    def __init__(self):
        self.ctx, self.owned, self.tensors, self.out = _ctx(), [], {}, None
        self.batch = self.event = self.call = None

    def own(self, x):
        self.owned.append(x)
        return x

    def bind(self, name, tensor):
        """A tensor of the program as a buffer of the runtime (the tensor keeps the memory)."""
        self.tensors[name] = tensor
        return self.own(self.ctx.import_buffer(tensor.data_ptr(), tensor.numel() * tensor.element_size()))

    def weight(self, t, N, K, gen):
        std, scale = (0.02 if K <= 8192 else 0.01), 1.0
        if t == "i2_s":
            scale = 1.2 / math.sqrt(K)
        return self.own(qmm.QuantWeight.from_ggml(self.ctx, TYPES[t][0], _ggml_blocks(t, N, K, std, gen), N, K, scale))

    def mul_mat(self, t, N, K, M, gen):
        return self.own(qmm.MulMat(self.ctx, self.weight(t, N, K, gen), M))

    def close(self):
        if self.event is not None:
            self.event.destroy()
        if self.batch is not None:
            self.batch.destroy()
        for x in reversed(self.owned):
            x.destroy()
        self.event = self.batch = None
        self.owned = []

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def _bits(v):
    return struct.unpack("<I", struct.pack("<f", float(v)))[0]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = _State()
    {"mul_mat": _prepare_mul_mat, "layer": _prepare_layer, "attention": _prepare_attention}[case["kind"]](s, case, gen)
    torch.cuda.synchronize()
    return s


def run(state):
    if state.call is not None:
        state.call()
    else:
        if state.event is not None:
            state.event.destroy()      # of this state's previous pass
        state.event = state.batch.replay()
    return state.out


def _prepare_mul_mat(s, c, gen):
    M, N, K = c["M"], c["N"], c["K"]
    mm = s.mul_mat(c["type"], N, K, M, gen)
    s.out = torch.zeros((M, N), device="cuda")
    x = s.bind("x", torch.randn((M, K), device="cuda", generator=gen))
    dst = s.bind("dst", s.out)
    if not c["replay"]:
        s.call = lambda: mm.run(x, dst, M)
        return
    s.batch = s.ctx.batch(64 + M)
    mm.record(s.batch, x, dst, M)
    s.batch.instantiate()


def _attention_push(c, n_q, mask_pitch):
    D, heads, kv = c["D"], c["heads"], c["kv_heads"]
    return [D, D, c["n_kv"], n_q, heads, kv, 0x11, int(mask_pitch > 0), 0, heads * D, D, 0, kv * D, D, 0, kv * D, D, 0, mask_pitch, 0,
            1, 0, _bits(1 / math.sqrt(D)), 0, 0, 0, 0, 0, 0, 0, 0]


def _causal_mask(n_q, n_kv):
    """[n_q][n_kv, padded]: position i sees the keys up to n_kv - n_q + i."""
    pitch = (n_kv + 63) // 64 * 64
    key = torch.arange(pitch, device="cuda").view(1, -1)
    last = torch.arange(n_kv - n_q, n_kv, device="cuda").view(-1, 1)
    return torch.where(key <= last, 0.0, float("-inf")).to(torch.float16)


def _prepare_attention(s, c, gen):
    D, n_q, n_kv = c["D"], c["n_q"], c["n_kv"]
    s.out = torch.zeros((n_q, c["heads"], D), device="cuda")
    q = s.bind("q", torch.randn((n_q, c["heads"] * D), device="cuda", generator=gen))
    k, v = (s.bind(name, torch.randn((n_kv, c["kv_heads"] * D), device="cuda", generator=gen).half()) for name in ("k", "v"))
    mask = _causal_mask(n_q, n_kv)
    scratch = s.own(s.ctx.buffer(16 << 20))
    s.batch = s.ctx.batch(8)
    s.batch.dispatch(s.ctx.kernel("ameva_flash_attn"), [q, k, v, s.bind("mask", mask), s.bind("out", s.out), scratch],
                     _attention_push(c, n_q, mask.shape[1]))
    s.batch.instantiate()


def _prepare_layer(s, c, gen):
    ctx, M, D, ff, n_kv, t, alt = s.ctx, c["M"], c["D"], c["ff"], c["n_kv"], c["type"], c["alt"]
    d, kv = c["heads"] * D, c["kv_heads"] * D
    eps = 1e-5

    def rows(name, width):
        return s.bind(name, torch.zeros((M, width), device="cuda"))

    def norm_weight(name):
        return s.bind(name, torch.empty(d, device="cuda").normal_(1.0, 0.1, generator=gen))

    # the residual stream some layers in: larger than what one layer adds
    x = s.bind("x", torch.empty((M, d), device="cuda").normal_(0.0, 4.0, generator=gen))
    norm1, norm2 = norm_weight("norm1"), norm_weight("norm2")
    k_cache, v_cache = (torch.randn((n_kv, kv), device="cuda", generator=gen).half() for _ in range(2))
    kc, vc = s.bind("k_cache", k_cache), s.bind("v_cache", v_cache)
    positions = torch.arange(n_kv - M, n_kv, device="cuda")
    pos, slots = s.bind("pos", positions.to(torch.int32)), s.bind("slots", positions.to(torch.int64))
    status = s.bind("status", torch.tensor([0, -1], device="cuda", dtype=torch.int32))
    mask = _causal_mask(M, n_kv)
    mb = s.bind("mask", mask)
    y, q, k, v, qr, kr, att = rows("y", d), rows("q", d), rows("k", kv), rows("v", kv), rows("qr", d), rows("kr", kv), rows("att", d)
    h, y2, gate, up, act = rows("h", d), rows("y2", d), rows("gate", ff), rows("up", ff), rows("act", ff)
    tmp = rows("tmp", d)
    out = torch.zeros((M, d), device="cuda")
    ob = s.bind("out", out)
    scratch = s.own(ctx.buffer(16 << 20))
    fused = t != "i2_s"            # the fused RMS norm + quantize and the one-row launches
    grouped = fused and M == 1
    b = s.batch = ctx.batch(1024 + 8 * M)

    def products(src, norm, normed, shapes, dsts):
        """RMS norm of src, then the products of `normed` with weights that share the type t."""
        if grouped:
            g = s.own(qmm.MulMatGroup(ctx, [s.weight(t, n, d, gen) for n in shapes], fused_quantize=False))
            g.record_rms_norm_quantize(b, src, normed, eps=eps, weight=norm)
            g.record(b, normed, dsts, quantize=False)
            return
        mms = [s.mul_mat(t, n, d, M, gen) for n in shapes]
        if fused:
            mms[0].record_rms_norm_quantize(b, src, normed, M, eps=eps, weight=norm)
        else:
            b.dispatch(ctx.kernel("ameva_rms_norm_f32"), [src, norm, normed], [M, d, _bits(eps), 1])
        for i, (mm, dst) in enumerate(zip(mms, dsts)):
            mm.record(b, normed, dst, M, quantize=not (fused and i == 0))

    def plus(tt, K, src, residual, dst):
        """dst = residual + product of src."""
        mm = s.mul_mat(tt, d, K, M, gen)
        if M == 1 and tt in ("q4_0", "q8_0", "q4_K"):
            mm.record(b, src, tmp, 1, epilogue=(qmm.EPILOGUE_ADD, residual, dst))
            return
        mm.record(b, src, tmp, M)
        b.dispatch(ctx.kernel("ameva_add_f32"), [tmp, residual, dst], [M, d, M])

    theta = _bits(10000.0 ** (-2.0 / D))
    if alt == t:
        products(x, norm1, y, [d, kv, kv], [q, k, v])
    else:
        products(x, norm1, y, [d, kv], [q, k])
        s.mul_mat(alt, kv, d, M, gen).record(b, y, v, M)
    for src, dst, n in ((q, qr, c["heads"]), (k, kr, c["kv_heads"])):
        w = n * D
        b.dispatch(ctx.kernel("ameva_rope"), [src, pos, pos, dst],
                   [D, n, M, 1, 0, D, w, w * M, 0, D, w, w * M, 0, 0, D, 1, 0, theta, _bits(1.0), _bits(0.0), _bits(1.0), 0, 0])
    for src, cache in ((kr, kc), (v, vc)):
        b.dispatch(ctx.kernel("ameva_set_rows"), [src, slots, status, cache],
                   [kv, M, 1, 1, 0, kv, kv * M, kv * M, 0, 2, 2 * M, 2 * M, 1, 1, 1, n_kv, 0, kv, kv * n_kv, kv * n_kv, 1, 0])
    b.dispatch(ctx.kernel("ameva_flash_attn"), [qr, kc, vc, mb, att, scratch], _attention_push(c, M, mask.shape[1]))
    plus(t, d, att, x, h)
    products(h, norm2, y2, [ff, ff], [gate, up])
    b.dispatch(ctx.kernel("ameva_swiglu_f32"), [gate, up, act], [M * ff])
    plus(alt, ff, act, h, ob)
    b.instantiate()
    s.out = {"out": out, "k_cache": k_cache, "v_cache": v_cache}
